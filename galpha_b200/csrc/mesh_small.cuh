// mesh_small.cuh -- the mesh stages from shifting to flipping as one launch,
// for small meshes (included by dt_mesh.cu, whose functors it runs).
//
// The launched stages of a mesh of a few thousand vertices are 60 to 90
// launches of 2 to 10 us of work and a dozen counter reads: a launch costs the
// host 2 us and a read 10 to 15 us of idle device, so the loops around the
// kernels, not the kernels, set the time.  Here one thread-block cluster runs
// all rounds of all stages: the phases are the launched kernels' functors over
// the same lists and counter words, separated by the cluster's hardware
// barrier (whose blocks are resident together by construction, so nothing
// spins), and the loop conditions are read on the device.  The mesh may differ
// from the launched stages' only where two launched runs may differ.  A call of
// 12,000 points takes 0.80 ms, with launched stages 1.12; 100,000 points 1.15 and
// 1.41 (sizes up to which each stage is run this way: kSmShiftV and below).
// What bounds it is the latency of the phases' gathers, and of one warp's chain
// of triangles in fake removal (0.12 of 0.23 ms at 1,000 points); 16 blocks of
// 512 threads hide it for up to some 10,000 items per phase.
//
// Every thread must take the same branches, so a counter word that decides one
// is read after a barrier and written only after the next one.
#pragma once

namespace galpha {

constexpr int kSmThreads = 512;   // per block: 128 registers per thread
constexpr int kSmFrWarps = 8;     // warps per block that remove fakes (shared memory)
constexpr int kSmPerBlock = 256;  // vertices per block

// The stored fans of a round are disjoint, fewer entries than triangle slots,
// so the long ones (over kMaxChain) find room, each at its own place, in an
// array of two edge records per slot that the mesh stages leave idle.
constexpr int kSmFanBytes = 42;
static_assert((size_t)kSmFanBytes * (kMaxChain + 1) >= fake_remove_smem(kMaxChain + 1) + 15, "a place holds its fan");
static_assert((size_t)kSmFanBytes * kMaxFanLong >= fake_remove_smem(kMaxFanLong) + 15, "a place holds its fan");
static_assert(kSmFanBytes <= 2 * sizeof(galphaEdgeInterval), "the array holds every place");

__device__ __noinline__ void fake_remove_long(const FakeRemoveArgs &a, int item, int d, unsigned char *mem, FrWarp &w)
{
    fake_remove_item(a, item, d, mem, w);
}

struct SmallMesh {
    // arrays of Ctx
    double2 *opos, *pos;
    int4 *tv, *tn, *fwd;
    int *epoch, *vote, *stamp, *freelist, *vtri, *vround, *anchor;
    int *list, *list2, *aux, *aux2, *inc;
    int8_t *vstate;
    Relink *rec;
    int2 *stage;      // fake runs: staged fan entries; flips: the triangles' states
    int *rec5;        // fake runs: records
    unsigned char *longfan;  // fans too long for shared memory, each at kSmFanBytes times its place in the store
    long long longfan_bytes;
    const unsigned long long *chash;
    unsigned cmask;
    Counters *ct;
    int N, F, V, cap, run_levels, round0, max_rounds;
    int rr0;          // words of r_rec taken before
    int from, to;     // stages to run (kSm*)
    int miss_limit;   // missing sites above which the launch ends before their insertion
};

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Whether the filters leave an edge of triangle t undecided.
__device__ __forceinline__ bool flip_undecided(const int4 *tv, const int4 *tn, const double2 *pos, int t)
{
    const int4 v = tv[t];
    if (v.x < 0) return false;
    const int4 n = tn[t];
    bool hard = false;
    for (int i = 0; i < 3; i++) {
        const int e = geti(n, i);
        if (e < 0) continue;
        int n64 = 0;
        hard |= incircle_fast(pos[geti(v, p1(i))], pos[geti(v, m1(i))], pos[geti(v, i)],
                              pos[geti(tv[dtri(e)], dori(e))], &n64) == 2;
    }
    return hard;
}

__global__ void __launch_bounds__(kSmThreads, 1) k_mesh_small(const SmallMesh m)
{
    extern __shared__ __align__(16) unsigned char sm_mem[];
    __shared__ FrWarp s_fr[kSmFrWarps];
    Counters *const ct = m.ct;
    unsigned cta_u, ncta_u;
    asm("mov.u32 %0, %cluster_ctarank;" : "=r"(cta_u));
    asm("mov.u32 %0, %cluster_nctarank;" : "=r"(ncta_u));
    const int cta = (int)cta_u, ncta = (int)ncta_u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nthr = ncta * kSmThreads, nwarp = nthr / 32;
    const int tid = cta * kSmThreads + (int)threadIdx.x;
    // irregular work (fan walks, point location, ear clipping) is dealt to the
    // warps first and to their lanes last: a short list then has few active
    // lanes per warp, which do not wait for one another's longer walks
    const int sid = lane * nwarp + warp * ncta + cta;
    const bool lead = tid == 0;
    auto each = [&](int n, auto f) {
        for (int i = tid; i < n; i += nthr) f(i);
    };
    auto spread = [&](int n, auto f) {
        for (int i = sid; i < n; i += nthr) f(i);
    };
    auto rd = [](const int *p) { return *(const volatile int *)p; };
    auto rg = [](int k) { return k % kRing; };
    int round = m.round0, rr = m.rr0;             // operation round ids, relink-record words
    int bad = 0;                                  // uniform: the detail of a failure, 0 if none
    int next = m.from;                            // first stage not run
    int shift_rounds = 0, missing_rounds = 0, flip_rounds = 0;
    int *const aux = m.aux, *const aux2 = m.aux2;

    // broken links (links_result) reach no stage
    if (next == kSmShift && (rd(&ct->err) || rd(&ct->nhull) != m.F)) bad = -1;
    if (next == kSmShift && !bad) {
        if (lead) ct->sm_ns[0] = global_ns();
        {
            int8_t *cand = (int8_t *)m.list2;
            int *drop = m.list2 + ((m.V + 1023) >> 2) + 256;
            const int nt = rd(&ct->ntris);
            each(m.V, ShiftCandidates{m.vstate, cand, drop});
            cluster_barrier();
            for (int it = 0; !bad; it++) {
                int *cur = it & 1 ? aux : m.list, *prev = it & 1 ? m.list : aux;
                int *curn = &ct->r_drop[rg(it)];
                if (it == 0) each(nt, ShiftCheckTris{m.tv, m.pos, m.opos, cand, drop, cur, curn, ct});
                else
                    spread(rd(&ct->r_drop[rg(it - 1)]),
                           ShiftCheckFans{m.tv, m.tn, m.vtri, m.pos, m.opos, cand, prev, drop, cur, curn, ct});
                cluster_barrier();
                const int n = rd(curn);
                each(n, ShiftDropList{cur, cand, drop, aux2, &ct->sh_total, m.N, ct});
                if (lead) ct->r_drop[rg(it + kRing / 2)] = 0;
                cluster_barrier();
                shift_rounds++;
                if (n == 0) break;
                if (shift_rounds >= m.max_rounds) bad = 301;
            }
            each(m.V, ShiftCommit{cand, m.pos, m.opos, m.vstate, m.vround});
            cluster_barrier();
        }
        const int ndrop = rd(&ct->sh_total);
        for (int k = 2; !bad; k++) {
            int *waiting = &ct->r_wait[rg(k)];
            spread(ndrop, ShiftRoundList{ShiftRound{m.tv, m.tn, m.pos, m.opos, m.vstate, m.vround, m.vtri, k, waiting,
                                                    ct},
                                         aux2});
            if (lead) ct->r_wait[rg(k + kRing / 2)] = 0;
            cluster_barrier();
            shift_rounds++;
            if (rd(waiting) == 0) break;
            if (shift_rounds > m.max_rounds) bad = 302;
        }
        int left = rd(&ct->nbad);
        for (int it = 0; left > 0 && !bad; it++) {
            int *nsel = &ct->r_bad[rg(it)], *nrec = &ct->r_rec[rg(rr)];
            spread(ndrop, BadSelectList{BadSelect{m.tv, m.tn, m.vstate, m.vtri, m.list, nsel}, aux2});
            if (lead) {
                ct->r_bad[rg(it + kRing / 2)] = 0;
                ct->r_rec[rg(rr + kRing / 2)] = 0;
            }
            cluster_barrier();
            const int n = rd(nsel);
            if (n == 0) break;
            round++;
            spread(n, BadRemove{m.tv, m.tn, m.fwd, m.epoch, m.freelist, m.vtri, m.anchor, m.list, m.pos, m.vstate,
                                m.rec, nrec, round, m.N, ct});
            cluster_barrier();
            each(rd(nrec), Relinker{m.tn, m.fwd, m.epoch, m.rec, m.tv, m.vtri, round, ct});
            if (lead) ct->sm_stop = ct->err;
            cluster_barrier();
            rr++;
            left -= n;
            if (rd(&ct->sm_stop)) bad = -1;
            if (it > m.max_rounds) bad = 303;
        }
        next = kSmMissing;
    }
    bool many = false;
    if (next == kSmMissing && m.to >= kSmMissing && !bad) {
        if (lead) ct->sm_ns[1] = global_ns();
        each(m.N, CountState{m.vstate, VS_MISSING, m.list, ct});
        cluster_barrier();
        const int nmiss = rd(&ct->nmiss);
        int remaining = nmiss;
        many = nmiss > m.miss_limit;
        if (many) {  // left to the launched rounds, which list them again
            remaining = 0;
            cluster_barrier();
            if (lead) ct->nmiss = 0;
        }
        for (int it = 0; remaining > 0 && !bad; it++) {
            int *nrec = &ct->r_rec[rg(rr)], *done = &ct->r_mis[rg(it)];
            round++;
            spread(nmiss, MissingLocate{m.tv, m.tn, m.pos, m.opos, m.vtri, m.anchor, m.vstate, m.list, aux, aux2,
                                        m.list2, m.vote, m.N, ct});
            cluster_barrier();
            spread(nmiss, MissingInsert{m.tv, m.tn, m.fwd, m.epoch, m.freelist, m.vtri, m.vote, m.pos, m.opos,
                                        m.vstate, m.list, aux, aux2, m.rec, nrec, done, round, m.cap, ct});
            cluster_barrier();
            each(rd(nrec), Relinker{m.tn, m.fwd, m.epoch, m.rec, m.tv, m.vtri, round, ct});
            each(nmiss, VotesBack{m.vote, aux, aux2, m.list2});
            if (lead) {
                if (ct->nfree < 0) ct->nfree = 0;
                ct->r_mis[rg(it + kRing / 2)] = 0;
                ct->r_rec[rg(rr + kRing / 2)] = 0;
                ct->sm_stop = ct->err;
            }
            cluster_barrier();
            rr++;
            missing_rounds++;
            const int n = rd(done);
            remaining -= n;
            if (rd(&ct->sm_stop)) bad = -1;
            else if (n == 0 || missing_rounds > m.max_rounds) bad = 304;
        }
        if (!many) next = kSmBoundary;
    }
    if (next == kSmBoundary && m.to >= kSmBoundary && !bad) {
        if (lead) ct->sm_ns[2] = global_ns();
        int *fanoff = m.anchor, *fanlen = m.vround;
        int2 *fan = (int2 *)m.inc;
        int removed = 0;
        bool runs = true;
        for (int pass = 0, it = 0; removed < m.F && !bad; pass++) {
            if (pass > m.max_rounds / 4) {
                bad = 305;
                break;
            }
            const int nsub = pass == 0 ? m.run_levels : 1;
            int now = removed;
            for (int q = 0; q < nsub && !bad; q++, it++) {
                int *nsel = &ct->r_fk[rg(it)], *nfan = &ct->r_fan[rg(it)], *nrec = &ct->r_rec[rg(rr)];
                round++;
                if (runs) {
                    const int level = pass == 0 ? q : -1;
                    spread(m.F, FakeRunStage{m.tv, m.tn, m.vstate, m.vtri, m.N, level, m.stage, &ct->r_stage[rg(it)],
                                             m.rec5, ct});
                    cluster_barrier();
                    spread(m.F, FakeRunJoin{m.vstate, m.N, level, m.stage, m.rec5, m.list, fanoff, fanlen, fan, nsel,
                                            nfan, ct});
                } else {
                    spread(m.F, FakeSelect{m.tv, m.tn, m.vstate, m.vtri, m.list, fanoff, fanlen, fan, nsel, nfan, m.N,
                                           ct});
                }
                cluster_barrier();
                now = rd(&ct->fk_removed);  // changes only in the next selection
                const int n = rd(nsel);
                const FakeRemoveArgs fr{m.tv, m.tn, m.fwd, m.epoch, m.freelist, m.vtri, m.list, fanoff, fanlen, fan,
                                        m.pos, m.vstate, m.rec, nrec, aux, round, ct};
                if (warp < kSmFrWarps)
                    for (int item = warp * ncta + cta; item < n; item += kSmFrWarps * ncta) {
                        const int d = fanlen[item] & 0xffff;
                        if (d <= kMaxChain)
                            fake_remove_item(fr, item, kMaxChain, sm_mem + warp * fake_remove_smem(kMaxChain), s_fr[warp]);
                        __syncwarp();
                    }
                if (warp == 0)  // fans too long for the shared arrays
                    for (int item = cta; item < n; item += ncta) {
                        const int d = fanlen[item] & 0xffff;
                        if (d > kMaxChain) {
                            const long long at = ((long long)kSmFanBytes * fanoff[item] + 15) & ~15ll;
                            if (at + (long long)fake_remove_smem(d) <= m.longfan_bytes)
                                fake_remove_long(fr, item, d, m.longfan + at, s_fr[0]);
                            else if (lane == 0)
                                set_err(ct, GPUDT_ERR_TOPOLOGY, 76);  // the fans overlap: a broken mesh
                        }
                        __syncwarp();
                    }
                cluster_barrier();
                each(rd(nrec), Relinker{m.tn, m.fwd, m.epoch, m.rec, m.tv, m.vtri, round, ct});
                if (lead) {
                    const int ahead = rg(it + kRing / 2);
                    ct->r_fk[ahead] = 0;
                    ct->r_fan[ahead] = 0;
                    ct->r_stage[ahead] = 0;
                    ct->r_rec[rg(rr + kRing / 2)] = 0;
                    ct->sm_stop = ct->err;
                }
                cluster_barrier();
                rr++;
                if (rd(&ct->sm_stop)) bad = -1;
            }
            const bool none = now == removed;
            if (!bad && none && !runs) bad = 306;  // priority always removes one
            runs = !none;
            removed = now;
        }
        if (!bad) {
            const int ncand = rd(&ct->ncand);
            if (lead) ct->nlist = ct->nlist2 = 0;
            each(m.V, [&](int i) { m.stamp[i] = -1; });
            cluster_barrier();
            round++;
            spread(ncand, ReflexCheck{m.tv, m.tn, m.pos, m.vtri, aux, m.vstate, m.list, m.stamp, round, ct});
            cluster_barrier();
            int *win = &ct->nlist, *wout = &ct->nlist2, *lin = m.list, *lout = m.list2;
            int n = rd(win);  // reflex vertices: fill them in rounds
            for (int guard = 0; n > 0 && !bad; guard++) {
                if (guard > m.max_rounds) {
                    bad = 307;
                    break;
                }
                round++;
                spread(n, ConvexPropose{m.tv, m.tn, m.pos, m.vtri, lin, nullptr, m.vote, m.fwd, ct});
                cluster_barrier();
                spread(n, ConvexApply{m.tv, m.tn, m.vtri, m.freelist, m.stamp, lin, m.vote, m.fwd, lout, wout, m.cap,
                                      round, ct});
                cluster_barrier();
                const int left = rd(wout);
                each(n, ConvexReset{m.fwd, lin, m.vote});
                if (lead) {
                    *win = 0;  // the next round's output count
                    ct->sm_stop = ct->err;
                }
                cluster_barrier();
                int *t = win;
                win = wout;
                wout = t;
                t = lin;
                lin = lout;
                lout = t;
                n = left;
                if (rd(&ct->sm_stop)) bad = -1;
            }
            if (lead && ct->nfree < 0) ct->nfree = 0;
        }
        next = kSmFlip;
    }
    bool exact = false;
    if (next == kSmFlip && m.to >= kSmFlip && !bad) {
        if (lead) ct->sm_ns[3] = global_ns();
        const int nt = rd(&ct->ntris);
        int2 *st = m.stage;
        each(nt, FlipInit{m.tv, st, m.vote, m.list, &ct->r_act[0]});
        // Exact tests are arithmetic, some 80 us each on coordinates that are no
        // multiples of a power of two, and want the whole GPU when there are more
        // of them than threads here (a lattice of spacing 1/3: 8,100 points 177
        // us, now 85; 25,600 points 663, now 112): each thread looks at one
        // triangle of an even spread (2.5 us), and by their share the flips are
        // handed back to launches.
        if (nt > nthr) {
            const bool hard = flip_undecided(m.tv, m.tn, m.pos, (int)((long long)tid * nt / nthr));
            const unsigned b = __ballot_sync(0xffffffffu, hard);
            if (lane == 0 && b) atomicAdd(&ct->sm_hard, __popc(b));
        }
        cluster_barrier();
        exact = (long long)rd(&ct->sm_hard) * nt > (long long)nthr * nthr;
        if (exact && lead) ct->r_act[0] = 0;
    }
    if (next == kSmFlip && m.to >= kSmFlip && !bad && !exact) {
        int2 *st = m.stage;
        int2 *cands = (int2 *)m.inc;
        FlipCheck ck{m.tv, m.tn, m.pos, nullptr, st, m.vote, cands, nullptr, ct, m.chash, m.cmask};
        FlipApply ap{m.tv, m.tn, st, m.vote, nullptr, nullptr, cands, m.rec, 0, ct, false, nullptr, nullptr, 3ll * m.cap};
        FlipRelink rl{m.tn, st, m.rec, 0};
        const FlipReset rs{m.vote, cands};
        // one round: the whole cluster, or block 0 alone (by = its threads, sync its barrier)
        auto flips = [&](int k, int n, int first, int by, auto sync) {
            const int w = rg(k), w1 = rg(k + 1), ahead = rg(k + kRing / 2);
            ck.act = k & 1 ? m.list2 : m.list;
            ck.cand_n = &ct->r_cand[w];
            for (int i = first; i < n; i += by) ck(i);
            sync();
            const int nc = rd(&ct->r_cand[w]);
            ap.next = k & 1 ? m.list : m.list2;
            ap.next_n = &ct->r_act[w1];
            ap.cand_n = &ct->r_cand[w];
            ap.rec_n = &ct->r_frec[w];
            ap.stamp = rl.stamp = k + 1;
            for (int i = first; i < nc; i += by) ap(i);
            sync();
            const int nr = rd(&ct->r_frec[w]);
            for (int i = first; i < nr; i += by) rl(i);
            for (int i = first; i < nc; i += by) rs(i);
            if (lead) {
                ct->r_act[ahead] = 0;
                ct->r_cand[ahead] = 0;
                ct->r_frec[ahead] = 0;
            }
            sync();
        };
        int k = 0;
        for (;;) {
            int n = rd(&ct->r_act[rg(k)]);
            if (n == 0) break;
            if (k > m.max_rounds) {
                bad = 308;
                break;
            }
            if (n > kSmThreads) {
                flips(k, n, tid, nthr, [] { cluster_barrier(); });
                k++;
                continue;
            }
            cluster_barrier();  // every block has read the list's length before block 0 reuses its word
            if (cta == 0) {  // a short list: block 0 alone until it empties or grows again
                do {
                    flips(k, n, (int)threadIdx.x, kSmThreads, [] { __syncthreads(); });
                    k++;
                    n = rd(&ct->r_act[rg(k)]);
                } while (n > 0 && n <= 2 * kSmThreads && k <= m.max_rounds);
                if (lead) ct->tail_rounds = k;
            }
            cluster_barrier();
            k = rd(&ct->tail_rounds);
        }
        flip_rounds = k;
        next = kSmFlip + 1;
    }
    if (lead) {
        ct->sm_ns[next] = global_ns();
        ct->sm_next = next;
        ct->sm_rec = rr;
        ct->sm_round = round;
        if (shift_rounds) ct->sm_shift = shift_rounds;
        if (missing_rounds) ct->sm_missing = missing_rounds;
        if (flip_rounds) ct->sm_flip = flip_rounds;
        if (bad > 0) set_err(ct, GPUDT_ERR_NOCONVERGE, bad);
    }
}

constexpr size_t kSmSmem = kSmFrWarps * fake_remove_smem(kMaxChain);

// Launch of one cluster of `blocks` blocks; at: filled in for it.
static cudaLaunchConfig_t small_mesh_config(const Ctx &c, int blocks, cudaLaunchAttribute *at)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kSmThreads);
    cfg.dynamicSmemBytes = kSmSmem;
    cfg.stream = c.stream;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = blocks;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

static int small_mesh_blocks(int V)
{
    int blocks = 1;
    while (blocks < kSmMaxBlocks && blocks * kSmPerBlock < V) blocks *= 2;
    return blocks;
}

// A block takes a whole SM, so a mesh of over 2,048 vertices needs 16 free ones
// in one GPC, which a whole B200 has and a part of one need not: the device is
// asked once per handle, and where the mesh's cluster does not fit (or is
// larger than allowed) the stages run as launches of their own.
bool small_mesh_fits(Ctx &c)
{
    if (c.sm_fit < 0) {
        cudaFuncSetAttribute(k_mesh_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmSmem);
        const bool large =
            cudaFuncSetAttribute(k_mesh_small, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        int fit = large ? kSmMaxBlocks : 8;
        for (; fit > 0; fit /= 2) {
            cudaLaunchAttribute at[1];
            const cudaLaunchConfig_t cfg = small_mesh_config(c, fit, at);
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, k_mesh_small, &cfg) == cudaSuccess && clusters > 0) break;
        }
        cudaGetLastError();  // an answer "cannot" is no error of the call
        c.sm_fit = fit;
    }
    return small_mesh_blocks(c.V) <= std::min(c.sm_fit, c.sm_limit);
}

static int launch_mesh_small(Ctx &c, int from, int to)
{
    SmallMesh m{};
    m.opos = c.opos;
    m.pos = c.pos;
    m.tv = c.tv;
    m.tn = c.tn;
    m.fwd = c.fwd;
    m.epoch = c.epoch;
    m.vote = c.vote;
    m.stamp = c.stamp;
    m.freelist = c.freelist;
    m.vtri = c.vtri;
    m.vround = c.vround;
    m.anchor = c.anchor;
    m.list = c.list;
    m.list2 = c.list2;
    m.aux = c.aux;
    m.aux2 = c.aux2;
    m.inc = c.inc;
    m.vstate = c.vstate;
    m.rec = c.rec;
    m.stage = (int2 *)c.keys2;  // alpha-stage buffers, idle until the mesh is final
    m.rec5 = (int *)c.spectrum;
    m.longfan = (unsigned char *)c.edge_aos;  // idle until an alpha result is downloaded
    m.longfan_bytes = 2ll * c.cap_tris * (long long)sizeof(galphaEdgeInterval);
    m.chash = c.chash;
    m.cmask = c.cmask;
    m.ct = c.ctr;
    m.N = c.N;
    m.F = c.F;
    m.V = c.V;
    m.cap = c.cap_tris;
    m.run_levels = 1;
    while (m.run_levels < 6 && (1LL << (4 * m.run_levels)) < c.F) m.run_levels++;
    m.round0 = c.round_counter;
    m.rr0 = c.rec_round;
    m.max_rounds = c.max_rounds;
    m.from = from;
    m.to = to;
    m.miss_limit = kSmMissLimit;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = small_mesh_config(c, small_mesh_blocks(c.V), at);
    GALPHA_CUDA(cudaLaunchKernelEx(&cfg, k_mesh_small, m));
    count_launch();
    return GPUDT_OK;
}

// Runs the stages `from` .. `to` in one launch and one counter read; *next is
// the first stage that has not been run (to + 1; kSmMissing when there are too
// many missing sites; kSmFlip when there are too many exact tests).
int stage_small(Ctx &c, int from, int to, int *next)
{
    int r = launch_mesh_small(c, from, to);
    if (r) return r;
    r = read_counters(c);
    if (r) return r;
    const Counters &h = *c.hctr;
    c.round_counter = std::max(c.round_counter, h.sm_round);
    c.rec_round = h.sm_rec;
    *next = h.sm_next;
    if (from == kSmShift && h.sm_next == kSmShift && (r = links_result(c))) return r;
    if (h.err) return h.err;
    if (h.ntris > c.cap_tris) return GPUDT_ERR_NOMEM;
    for (int s = from; s < h.sm_next; s++) c.small_ms[s] = (float)((double)(h.sm_ns[s + 1] - h.sm_ns[s]) * 1e-6);
    if (from <= kSmShift) {
        c.st.shiftRounds = h.sm_shift;
        c.st.nBadShift = h.nbad;
    }
    if (from <= kSmMissing && h.sm_next > kSmMissing) {
        c.st.nMissing = h.nmiss;
        c.st.nDuplicates = h.ndup;
        c.st.missingRounds = h.sm_missing;
    }
    if (h.sm_next > kSmFlip) {
        c.st.nFlips = h.flips_total;
        c.st.flipRounds = h.sm_flip;
    }
    return GPUDT_OK;
}

}  // namespace galpha
