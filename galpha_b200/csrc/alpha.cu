// alpha.cu -- alpha spectrum and per-simplex intervals on the device.
//
// Stage map (reference -> here):
//   computeTriEdgeCount + exclusive_scan +          k_alpha_keys: the reference's ownership
//   computeEdgeTriMap (kernel.cu:138-217)           and numbering rule (offsets by look-back)
//   computeTriangleRo / computeEdgeRo /             k_alpha_keys: birth times in
//   processAttached (kernel.cu:219-358,             double-double (<= 1 ulp, certified),
//   predicates.h:1297-1444)                         slivers recomputed exactly; attached test
//                                                   filtered then exact (closed disc)
//   thrust::remove_if x2 (Alpha_Shapes_2D.cu:       k_alpha_keys: unattached edges compacted
//   276-281)                                        by the same look-back
//   thrust::sort_by_key (Alpha_Shapes_2D.cu:317)    radix_sort: LSD radix sort of the FP64
//                                                   bit patterns with an int payload
//   markSpectrum + sorT odd-even rounds +           k_mark_runs / k_resolve_runs: every run
//   CPU_insertion_sort (kernel.cu:785-1102,         of keys within 2 ulp is sorted with the
//   Alpha_Shapes_2D.cu:344-610)                     exact comparator on the device; exact
//                                                   ties share a rank
//   processSpectrum / remove_if / UpdateBackRefs    scan of "new rank" flags + k_scatter_ranks
//   (kernel.cu:360-401, Alpha_Shapes_2D.cu:483-512)
//   edgeIntervals / computeVertexIntervals          k_edge_intervals / k_vertex_intervals:
//   (kernel.cu:427-624)                             vertex min/max by atomics over edges
#include <cstdio>
#include <algorithm>
#include <vector>
#include "internal.cuh"
#include "exact.cuh"
#include "block_sort.cuh"

namespace galpha {

// ------------------------------------------------------------ double-double
struct dd {
    double h, l;
};

__device__ __forceinline__ dd dd_from_diff(double a, double b)
{
    dd r;
    two_sum(a, -b, r.h, r.l);
    return r;
}

__device__ __forceinline__ dd dd_mul(dd a, dd b)
{
    double p, e;
    two_prod(a.h, b.h, p, e);
    e = fma(a.h, b.l, e);
    e = fma(a.l, b.h, e);
    dd r;
    fast_two_sum(p, e, r.h, r.l);
    return r;
}

__device__ __forceinline__ dd dd_add(dd a, dd b)
{
    double s, e;
    two_sum(a.h, b.h, s, e);
    e += a.l + b.l;
    dd r;
    fast_two_sum(s, e, r.h, r.l);
    return r;
}

__device__ __forceinline__ dd dd_sub(dd a, dd b)
{
    b.h = -b.h;
    b.l = -b.l;
    return dd_add(a, b);
}

__device__ __forceinline__ double dd_div_to_double(dd a, dd b)
{
    double q1 = a.h / b.h;
    dd qb = dd_mul(dd{q1, 0.0}, b);
    dd r = dd_sub(a, qb);
    double q2 = r.h / b.h;
    return q1 + q2;
}

__device__ __forceinline__ dd dd_sqdist(double2 p, double2 q)
{
    dd dx = dd_from_diff(p.x, q.x), dy = dd_from_diff(p.y, q.y);
    return dd_add(dd_mul(dx, dx), dd_mul(dy, dy));
}

// Edge birth time (|pq|/2)^2.
__device__ __forceinline__ double rho_edge(double2 p, double2 q)
{
    dd s = dd_sqdist(p, q);
    return (s.h + s.l) * 0.25;
}

// Triangle birth time R^2 = abc / (4 ar^2); *sliver set when ar is too
// cancelled for the double-double evaluation to certify 1 ulp.
__device__ __forceinline__ double rho_tri(double2 A, double2 B, double2 C, bool *sliver)
{
    dd a = dd_sqdist(A, B), b = dd_sqdist(B, C), c = dd_sqdist(C, A);
    dd N = dd_mul(dd_mul(a, b), c);
    dd ux = dd_from_diff(B.x, A.x), vy = dd_from_diff(C.y, A.y);
    dd vx = dd_from_diff(C.x, A.x), uy = dd_from_diff(B.y, A.y);
    dd P1 = dd_mul(ux, vy), P2 = dd_mul(vx, uy);
    dd ar = dd_sub(P1, P2);
    double mag = fabs(P1.h) + fabs(P2.h);
    *sliver = !(fabs(ar.h) >= ldexp(mag, -48));
    dd D = dd_mul(ar, ar);
    D.h *= 4.0;
    D.l *= 4.0;
    return dd_div_to_double(N, D);
}

// ------------------------------------------------------------------ kernels
// The owned edges (mask `und`) of triangle t that the filter leaves undecided:
// returns the mask of those that are unattached.  A call that reads its operands
// again, after the loop over a thread's triangles: what lives across a call, and
// what the exact test takes by address, is kept in local memory, and in that loop
// every triangle stored and loaded it there (more L1 sectors than its gathers).
__device__ __noinline__ unsigned attached_hard(const int4 *gv, const int4 *cn, const double2 *P, long long t,
                                               unsigned und, Counters *ct)
{
    const int4 g = gv[t], n = cn[t];
    unsigned un = 0;
    for (int i = 0; i < 3; i++) {
        if (!((und >> i) & 1u)) continue;
        const double2 pa = P[geti(g, p1(i))], pb = P[geti(g, m1(i))], pk = P[geti(g, i)];
        const double qa[2] = {pa.x, pa.y}, qb[2] = {pb.x, pb.y}, qk[2] = {pk.x, pk.y};
        int att = attached_filter(qa, qb, qk);
        if (att == 2) {
            atomicAdd(&ct->exact_attached, 1ull);
            att = attached_exact(qa, qb, qk);
        }
        const int nb = geti(n, i);
        if (att == 0 && nb >= 0) {
            const double2 po = P[((const int *)gv)[4ll * dtri(nb) + dori(nb)]];
            const double qo[2] = {po.x, po.y};
            att = attached_filter(qa, qb, qo);
            if (att == 2) {
                atomicAdd(&ct->exact_attached, 1ull);
                att = attached_exact(qa, qb, qo);
            }
        }
        if (att == EXACT_OVERFLOW) set_err(ct, GPUDT_ERR_EXACT, 100);
        if (!att) un |= 1u << i;
    }
    return un;
}

// Triangle keys, edge numbering, attached tests and edge keys in one pass over
// the triangles.  A block takes the next tile of kAkTile triangles by ticket,
// computes their birth times, which edges they own and which of those are
// unattached (their birth times stay in shared memory), and finds the edges
// and the unattached edges of all earlier tiles by decoupled look-back; then
// it writes the tile's edges and edge keys at their places.  The loads are a
// triangle's three records, its corners and, for an owned edge its own corner
// leaves unattached, the corner across it; bound by the latency of those
// gathers (issue slots 40 % busy at 32 warps per SM, which the registers of the
// double-double arithmetic allow), so a round's records are loaded one round
// ahead, and by the wait for earlier tiles: 4 triangles per thread took 0.57
// ms at 8.0 M triangles, 2 took 0.64, 1 took 0.75, 8 by blocks of 128 took
// 0.80 (longer chains ahead of the tiles that wait); 0.48 since the exact tests
// are made after the loop.  Up to kAkFew triangles per SM (151,552 on 148)
// there are too few tiles of four to fill the GPU and one per thread is used
// (2,000 triangles: 20 us with four, 7 with one).  As five launches (edge
// counts, a scan, keys, a scan over the edges, edge keys from a second gather)
// it took 0.77 ms, and a counter read between the first and the third.
// A status word holds kind (bits 63-62), the edges (61-31) and the unattached
// edges (30-0) of its tile or of all tiles up to it; fewer than 2^31 edges.
constexpr int kAkSpinLimit = 1 << 22;
constexpr int kAkThreads = 256, kAkItemsMany = 4;
constexpr int kAkFew = 4 * kAkThreads;  // triangles per SM: its resident blocks, one each
constexpr unsigned long long kAkAgg = 1ull << 62, kAkInc = 2ull << 62, kAkVal = (1ull << 62) - 1;

struct AlphaKeysArgs {
    const int4 *cv, *cn;
    const int4 *gv;  // the triangles with the ids that index P
    const double2 *P;
    int nT;
    int *e_off;
    unsigned long long *keys;
    int *vals;
    int *edges;     // enc(tIndex, vOpp)
    int *edge_ro;   // 0 for attached edges
    int *slivers;
    unsigned long long *status;  // [tiles], zero; then the ticket
    int tiles;
    int2 *pt;       // [N] vertex intervals, started here
    int N;
    Counters *ct;
};

template <int kAkItems>
__global__ void __launch_bounds__(kAkThreads, 4) k_alpha_keys(AlphaKeysArgs A)
{
    constexpr int kAkTile = kAkThreads * kAkItems;
    for (int i = blockIdx.x * kAkThreads + threadIdx.x; i < A.N; i += gridDim.x * kAkThreads)
        A.pt[i] = make_int2(-1, -1);
    __shared__ double s_rho[3 * kAkTile];  // birth time of edge i of the tile's triangle j at [i][j]
    __shared__ int s_part[kAkItems * (kAkThreads / 32)];
    __shared__ int s_tile;
    __shared__ unsigned long long s_excl;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd((int *)(A.status + A.tiles), 1);
    __syncthreads();
    const int tile = s_tile;
    unsigned flags[kAkItems];  // bits 0-2 owned edges, 3-5 unattached ones, 6-8 undecided ones
    int incl[kAkItems], cnt[kAkItems];  // owned | unattached << 16
    const long long t0 = (long long)tile * kAkTile + threadIdx.x;
    int4 v, n, g;  // the next triangle's records, loaded one round ahead
    if (t0 < A.nT) {
        v = A.cv[t0];
        n = A.cn[t0];
        g = A.gv[t0];
    }
#pragma unroll 1
    for (int u = 0; u < kAkItems; u++) {
        const int j = u * kAkThreads + threadIdx.x;
        const long long t = t0 + u * kAkThreads;
        unsigned f = 0;
        if (t < A.nT) {
            const double2 Q[3] = {A.P[g.x], A.P[g.y], A.P[g.z]};
            // the corner across each owned edge: one word of its triangle, in
            // flight with the corners
            int nb[3], opp[3];
#pragma unroll
            for (int i = 0; i < 3; i++) {
                nb[i] = geti(n, i);
                const bool own = geti(v, p1(i)) < geti(v, m1(i)) || nb[i] == -1;
                f |= own ? 1u << i : 0u;
                opp[i] = own && nb[i] >= 0 ? ((const int *)A.gv)[4ll * dtri(nb[i]) + dori(nb[i])] : -1;
            }
            if (u + 1 < kAkItems && t + kAkThreads < A.nT) {
                v = A.cv[t + kAkThreads];
                n = A.cn[t + kAkThreads];
                g = A.gv[t + kAkThreads];
            }
            double2 O[3];
#pragma unroll
            for (int i = 0; i < 3; i++) O[i] = opp[i] >= 0 ? A.P[opp[i]] : make_double2(0.0, 0.0);
            bool sl;
            const double r = rho_tri(Q[0], Q[1], Q[2], &sl);
            A.keys[1 + t] = (unsigned long long)__double_as_longlong(r);
            A.vals[1 + t] = (int)t;
            if (sl) A.slivers[atomicAdd(&A.ct->al_sliver, 1)] = (int)t;
#pragma unroll
            for (int i = 0; i < 3; i++) {
                if (!((f >> i) & 1u)) continue;
                const double2 pa = Q[p1(i)], pb = Q[m1(i)], pk = Q[i], po = O[i];
                const double qa[2] = {pa.x, pa.y}, qb[2] = {pb.x, pb.y}, qk[2] = {pk.x, pk.y};
                int att = attached_filter(qa, qb, qk);
                if (att == 0 && opp[i] >= 0) {
                    const double qo[2] = {po.x, po.y};
                    att = attached_filter(qa, qb, qo);
                }
                f |= (att == 0 ? 8u : att == 2 ? 64u : 0u) << i;
                if (att != 1) s_rho[i * kAkTile + j] = rho_edge(pa, pb);
            }
        }
#pragma unroll
        for (int q = 0; q < kAkItems; q++)
            if (q == u) flags[q] = f;  // (registers have no run-time index)
    }
#pragma unroll
    for (int u = 0; u < kAkItems; u++) {
        if (flags[u] >> 6) flags[u] |= attached_hard(A.gv, A.cn, A.P, t0 + u * kAkThreads, flags[u] >> 6, A.ct) << 3;
    }
#pragma unroll
    for (int u = 0; u < kAkItems; u++) {
        const unsigned f = flags[u];
        int x = __popc(f & 7u) | (__popc(f & 56u) << 16);
        cnt[u] = x;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_part[u * (kAkThreads / 32) + w] = x;
        incl[u] = x;
    }
    __syncthreads();
    if (w == 0) {
        constexpr int kParts = kAkItems * (kAkThreads / 32);
        static_assert(kParts <= 32, "one warp scans the partial sums of a tile");
        const int v = lane < kParts ? s_part[lane] : 0;
        int x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane < kParts) s_part[lane] = x - v;
        const int tot = __shfl_sync(0xffffffffu, x, 31);
        const unsigned long long mine = ((unsigned long long)(tot & 0xffff) << 31) | (unsigned)(tot >> 16);
        unsigned long long acc = 0;
        if (tile > 0) {
            volatile unsigned long long *st = A.status;
            if (lane == 0) st[tile] = kAkAgg | mine;
            bool bad = false;
            for (int j = tile - 1;; j -= 32) {
                const int idx = j - lane;
                unsigned long long wd = kAkInc;  // before tile 0: nothing to add
                for (int spins = 0; idx >= 0 && ((wd = st[idx]) >> 62) == 0; spins++) {
                    if (spins > kAkSpinLimit) {
                        bad = true;
                        break;
                    }
                    __nanosleep(32);
                }
                bad = __any_sync(0xffffffffu, bad);
                if (bad) break;
                const unsigned inc = __ballot_sync(0xffffffffu, (wd >> 62) == 2);
                const int first = inc ? __ffs(inc) - 1 : 31;  // lanes up to the nearest inclusive count
                unsigned long long add = lane <= first && idx >= 0 ? wd & kAkVal : 0ull;
                for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
                acc += add;
                if (inc) break;
            }
            if (bad && lane == 0) set_err(A.ct, GPUDT_ERR_NOCONVERGE, 96);
        }
        if (lane == 0) {
            ((volatile unsigned long long *)A.status)[tile] = kAkInc | (acc + mine);
            s_excl = acc;
            if (tile == A.tiles - 1) {
                A.ct->al_edges = (int)((acc + mine) >> 31);
                A.ct->al_unatt = (int)((acc + mine) & 0x7fffffffu);
            }
        }
    }
    __syncthreads();
    const int e0 = (int)(s_excl >> 31), k0 = 1 + A.nT + (int)(s_excl & 0x7fffffffu);
#pragma unroll
    for (int u = 0; u < kAkItems; u++) {
        const int j = u * kAkThreads + threadIdx.x;
        const long long t = (long long)tile * kAkTile + j;
        if (t >= A.nT) continue;
        const int at = s_part[u * (kAkThreads / 32) + w] + incl[u] - cnt[u];
        int e = e0 + (at & 0xffff), k = k0 + (at >> 16);
        A.e_off[t] = e;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            if (!((flags[u] >> i) & 1u)) continue;
            A.edges[e] = enc((int)t, i);
            if ((flags[u] >> i) & 8u) {
                A.keys[k] = (unsigned long long)__double_as_longlong(s_rho[i * kAkTile + j]);
                A.vals[k++] = A.nT + e;
            } else {
                A.edge_ro[e] = 0;
            }
            e++;
        }
    }
}

struct SliverKeys {
    const int4 *cv;  // the triangles with the ids that index P
    const double2 *P;
    const int *slivers;
    unsigned long long *keys;
    Counters *ct;
    __device__ void operator()(long long ii) const
    {
        int t = slivers[ii];
        int4 v = cv[t];
        double p[6] = {P[v.x].x, P[v.x].y, P[v.y].x, P[v.y].y, P[v.z].x, P[v.z].y};
        double r = rho_rounded_exact(3, p);
        if (r != r) set_err(ct, GPUDT_ERR_EXACT, 101);
        keys[1 + t] = (unsigned long long)__double_as_longlong(r);
    }
};

// --------------------------------------------------------- ranks and runs
__device__ __forceinline__ bool near_equal(unsigned long long ka, unsigned long long kb)
{
    // kb >= ka (sorted); keys carry <= 1 ulp of error each
    double a = __longlong_as_double((long long)ka), b = __longlong_as_double((long long)kb);
    double u = __longlong_as_double((long long)kb + 1) - b;  // ulp of the positive key b
    return (b - a) <= 2.0 * u;
}

// nr[i] = 1 when entry i certainly starts a new rank.  Links within 2 ulp are
// listed for one exact comparison each.
struct MarkRuns {
    const unsigned long long *keys;
    int *nr;
    int *unc;
    int n;
    Counters *ct;
    const int *seg;  // set of each entry (batched stage) or nullptr
    __device__ void operator()(long long ii) const
    {
        int i = (int)ii;
        if (i == 0) {
            nr[0] = 0;
            return;
        }
        if (i >= 2 && (!seg || seg[i] == seg[i - 1]) && near_equal(keys[i - 1], keys[i])) {
            nr[i] = 0;
            int k = atomicAdd(&ct->al_unc, 1);
            unc[k] = i;
        } else {
            nr[i] = 1;
        }
    }
};

__device__ __forceinline__ void entry_points(int val, int nT, const int4 *cv, const int *edges,
                                             const double2 *P, int *kind, double *p)
{
    if (val < nT) {
        int4 v = cv[val];
        double2 a = P[v.x], b = P[v.y], c = P[v.z];
        p[0] = a.x; p[1] = a.y; p[2] = b.x; p[3] = b.y; p[4] = c.x; p[5] = c.y;
        *kind = 3;
    } else {
        const int E = edges[val - nT];
        const int4 g = cv[dtri(E)];  // cv: the triangles with the ids that index P
        double2 a = P[geti(g, p1(dori(E)))], b = P[geti(g, m1(dori(E)))];
        p[0] = a.x; p[1] = a.y; p[2] = b.x; p[3] = b.y;
        *kind = 2;
    }
}

__device__ __forceinline__ int exact_cmp_vals(int va, int vb, int nT, const int4 *cv, const int *edges,
                                              const double2 *P)
{
    int ka, kb;
    double pa[6], pb[6];
    entry_points(va, nT, cv, edges, P, &ka, pa);
    entry_points(vb, nT, cv, edges, P, &kb, pb);
    return compare_rho_exact(ka, pa, kb, pb);
}

// One exact comparison per uncertain adjacent pair (parallel over pairs): a
// smaller left value starts a new rank, an exact tie shares the rank, and an
// order violation sends the whole run to k_resolve (rare: it needs two distinct
// values within one ulp whose keys rounded the wrong way).  Without slowflag
// the runs are only counted: the caller starts over when there is one.
struct ExactAdjacent {
    const unsigned long long *keys;
    const int *vals;
    int *nr, *slow, *slowflag;
    const int *unc;
    const int4 *cv;
    const int *edges;
    const double2 *P;
    int nT;
    Counters *ct;
    const int *seg;
    __device__ void operator()(long long ii) const
    {
        if (ct->err) return;  // a sort that gave up leaves entries that name no simplex
        int i = unc[ii];
        int cmp = exact_cmp_vals(vals[i - 1], vals[i], nT, cv, edges, P);
        atomicAdd(&ct->exact_compares, 1ull);
        if (cmp == EXACT_OVERFLOW) {
            set_err(ct, GPUDT_ERR_EXACT, 110);
            return;
        }
        if (cmp < 0) {
            nr[i] = 1;
        } else if (cmp == 0) {
            nr[i] = 0;
            atomicAdd(&ct->nties, 1);
        } else {
            int s = i - 1;
            if (!slowflag) {
                atomicAdd(&ct->al_slow, 1);
                return;
            }
            while (s >= 2 && (!seg || seg[s - 1] == seg[s]) && near_equal(keys[s - 1], keys[s])) s--;
            if (atomicCAS(&slowflag[s], 0, 1) == 0) {
                int k = atomicAdd(&ct->al_slow, 1);
                slow[k] = s;
            }
        }
    }
};

// Rare path: a run with an order violation is re-sorted with the exact
// comparator and its rank-start flags recomputed: one thread per run of at
// most kThreadRun entries (insertion sort), one block per longer run
// (k_resolve_long: merge sort), and a run longer than Ctx::block_run by many
// blocks, one launch per merge level (k_merge_level; a lattice of
// non-dyadic spacing gives runs of millions of near-equal radii).
constexpr int kThreadRun = 512;
struct ResolveRuns {
    unsigned long long *keys;
    int *vals, *nr;
    const int *runs;
    const int4 *cv;
    const int *edges;
    const double2 *P;
    int n, nT;
    Counters *ct;
    const int *seg;
    int *longs;  // runs longer than kThreadRun, for k_resolve_long (count in ct->nlong)
    __device__ void operator()(long long ii) const
    {
        int s = runs[ii];
        int e = s;
        while (e + 1 < n && (!seg || seg[e] == seg[e + 1]) && near_equal(keys[e], keys[e + 1])) {
            e++;
            if (e - s >= kThreadRun) {
                longs[atomicAdd(&ct->nlong, 1)] = s;
                return;
            }
        }
        for (int a = s + 1; a <= e; a++) {
            unsigned long long kc = keys[a];
            int vc = vals[a];
            int b = a - 1;
            for (; b >= s; b--) {
                int cmp = exact_cmp_vals(vals[b], vc, nT, cv, edges, P);
                if (cmp == EXACT_OVERFLOW) {
                    set_err(ct, GPUDT_ERR_EXACT, 111);
                    return;
                }
                if (cmp <= 0) break;
                keys[b + 1] = keys[b];
                vals[b + 1] = vals[b];
            }
            keys[b + 1] = kc;
            vals[b + 1] = vc;
        }
        for (int a = s + 1; a <= e; a++) {
            int cmp = exact_cmp_vals(vals[a - 1], vals[a], nT, cv, edges, P);
            if (cmp == EXACT_OVERFLOW) {
                set_err(ct, GPUDT_ERR_EXACT, 112);
                return;
            }
            nr[a] = cmp != 0 ? 1 : 0;
        }
    }
};

// Order of two spectrum entries: by key where the keys are more than 2 ulp
// apart (each carries at most 1 ulp of error), else exactly.
__device__ __forceinline__ int cmp_entries(unsigned long long ka, int va, unsigned long long kb, int vb, int nT,
                                           const int4 *cv, const int *edges, const double2 *P)
{
    if (ka < kb && !near_equal(ka, kb)) return -1;
    if (kb < ka && !near_equal(kb, ka)) return 1;
    return exact_cmp_vals(va, vb, nT, cv, edges, P);
}

// One block per long run starting at runs[blockIdx.x]: the run's end by
// block-wide scans, a stable bottom-up merge sort of (keys, vals)[s..e] with
// the exact comparator (each thread merges a share of the outputs from a
// merge-path split found by binary search; ties take the left run first),
// through (tk, tv)[s..e] as the second buffer, then the rank-start flags.
constexpr int kLongThreads = 256;
__global__ void __launch_bounds__(kLongThreads) k_resolve_long(unsigned long long *keys, int *vals, int *nr,
                                                               unsigned long long *tk, int *tv, const int *runs,
                                                               const int4 *cv, const int *edges, const double2 *P,
                                                               int n, int nT, Counters *ct, const int *seg,
                                                               int block_run, int2 *huge)
{
    __shared__ int red[kLongThreads / 32];
    __shared__ int s_end;
    const int s = runs[blockIdx.x];
    if (threadIdx.x == 0) s_end = n - 1;
    __syncthreads();
    // the run ends before the first j > s that is not linked to j - 1
    for (long long w0 = s + 1; w0 < n; w0 += kLongThreads) {
        const long long j = w0 + threadIdx.x;
        const bool brk = j < n && (!((!seg || seg[j - 1] == seg[j]) && near_equal(keys[j - 1], keys[j])));
        int m = __reduce_min_sync(0xffffffffu, brk ? (int)j : n);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        __syncthreads();
        m = red[0];
        for (int q = 1; q < kLongThreads / 32; q++) m = min(m, red[q]);
        __syncthreads();
        if (m < n) {
            if (threadIdx.x == 0) s_end = m - 1;
            break;
        }
    }
    __syncthreads();
    const int e = s_end, L = e - s + 1;
    if (L > block_run) {  // left to the multi-block merge
        if (threadIdx.x == 0) huge[atomicAdd(&ct->nhuge, 1)] = make_int2(s, L);
        return;
    }
    bool bad = false;
    unsigned long long *sk = keys + s, *dk = tk + s;
    int *sv = vals + s, *dv = tv + s;
    const int chunk = (L + kLongThreads - 1) / kLongThreads;
    for (int w = 1; w < L; w <<= 1) {
        const int o0 = min(L, (int)threadIdx.x * chunk), o1 = min(L, o0 + chunk);
        for (int pos = o0; pos < o1;) {
            const int lo = pos / (2 * w) * (2 * w), mid = min(L, lo + w), hi = min(L, lo + 2 * w);
            const int na = mid - lo, nb = hi - mid;
            const int k0 = pos - lo, kend = min(o1, hi) - lo;
            // merge-path split of diagonal k0: i elements of A before it
            int a0 = max(0, k0 - nb), a1 = min(k0, na);
            while (a0 < a1) {
                const int m = (a0 + a1) >> 1;
                int c = cmp_entries(sk[lo + m], sv[lo + m], sk[mid + k0 - m - 1], sv[mid + k0 - m - 1], nT, cv, edges, P);
                if (c == EXACT_OVERFLOW) {
                    bad = true;
                    c = 0;
                }
                if (c <= 0) a0 = m + 1;
                else a1 = m;
            }
            int i = a0, j = k0 - a0;
            for (int k = k0; k < kend; k++) {
                bool takeA = i < na;
                if (takeA && j < nb) {
                    int c = cmp_entries(sk[lo + i], sv[lo + i], sk[mid + j], sv[mid + j], nT, cv, edges, P);
                    if (c == EXACT_OVERFLOW) {
                        bad = true;
                        c = 0;
                    }
                    takeA = c <= 0;
                }
                const int src = takeA ? lo + i++ : mid + j++;
                dk[lo + k] = sk[src];
                dv[lo + k] = sv[src];
            }
            pos = lo + kend;
        }
        __syncthreads();  // every output of this level written before the next reads it
        unsigned long long *t1 = sk;
        sk = dk;
        dk = t1;
        int *t2 = sv;
        sv = dv;
        dv = t2;
    }
    if (sk != keys + s)  // the last level wrote the second buffer
        for (int k = threadIdx.x; k < L; k += kLongThreads) {
            keys[s + k] = sk[k];
            vals[s + k] = sv[k];
        }
    __syncthreads();
    for (int a = s + 1 + threadIdx.x; a <= e; a += kLongThreads) {
        int cmp = exact_cmp_vals(vals[a - 1], vals[a], nT, cv, edges, P);
        if (cmp == EXACT_OVERFLOW) {
            bad = true;
            cmp = 1;
        }
        nr[a] = cmp != 0 ? 1 : 0;
    }
    if (bad) set_err(ct, GPUDT_ERR_EXACT, 111);
}

// One merge level of the multi-block exact sort of a run of L entries:
// sorted blocks of w entries are merged pairwise from (sk, sv) into (dk, dv).
// Thread t writes outputs [t*kMergeChunk, (t+1)*kMergeChunk): for each pair
// of blocks its outputs fall in, it finds where its first output's merge path
// crosses the pair by binary search (ties take the left block first, so the
// sort is stable), then merges.
constexpr int kMergeChunk = 16;
__global__ void __launch_bounds__(256) k_merge_level(const unsigned long long *__restrict__ sk,
                                                     const int *__restrict__ sv, unsigned long long *__restrict__ dk,
                                                     int *__restrict__ dv, int L, int w, const int4 *cv,
                                                     const int *edges, const double2 *P, int nT, Counters *ct)
{
    const long long o0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * kMergeChunk;
    if (o0 >= L) return;
    const long long o1 = min((long long)L, o0 + kMergeChunk);
    bool bad = false;
    // the chunk may span several pairs of blocks while 2w < kMergeChunk
    for (long long pos = o0; pos < o1;) {
        const int lo = (int)(pos / (2ll * w) * (2ll * w));
        const int mid = (int)min((long long)L, (long long)lo + w);
        const int hi = (int)min((long long)L, (long long)lo + 2ll * w);
        const int na = mid - lo, nb = hi - mid;
        const int k0 = (int)pos - lo, kend = (int)min((long long)hi, o1) - lo;
        int a0 = max(0, k0 - nb), a1 = min(k0, na);
        while (a0 < a1) {
            const int m = (a0 + a1) >> 1;
            int c = cmp_entries(sk[lo + m], sv[lo + m], sk[mid + k0 - m - 1], sv[mid + k0 - m - 1], nT, cv, edges,
                                P);
            if (c == EXACT_OVERFLOW) {
                bad = true;
                c = 0;
            }
            if (c <= 0) a0 = m + 1;
            else a1 = m;
        }
        int i = a0, j = k0 - a0;
        for (int k = k0; k < kend; k++) {
            bool takeA = i < na;
            if (takeA && j < nb) {
                int c = cmp_entries(sk[lo + i], sv[lo + i], sk[mid + j], sv[mid + j], nT, cv, edges, P);
                if (c == EXACT_OVERFLOW) {
                    bad = true;
                    c = 0;
                }
                takeA = c <= 0;
            }
            const int src = takeA ? lo + i++ : mid + j++;
            dk[lo + k] = sk[src];
            dv[lo + k] = sv[src];
        }
        pos = lo + kend;
    }
    if (bad) set_err(ct, GPUDT_ERR_EXACT, 114);
}

// Rank-start flags of a sorted run [s, s + L): an entry starts a new rank
// unless it equals its left neighbour exactly.
struct RunFlags {
    const int *vals;
    int *nr;
    const int4 *cv;
    const int *edges;
    const double2 *P;
    int s, nT;
    Counters *ct;
    __device__ void operator()(long long ii) const
    {
        const int a = s + 1 + (int)ii;
        int cmp = exact_cmp_vals(vals[a - 1], vals[a], nT, cv, edges, P);
        if (cmp == EXACT_OVERFLOW) {
            set_err(ct, GPUDT_ERR_EXACT, 115);
            cmp = 1;
        }
        nr[a] = cmp != 0 ? 1 : 0;
    }
};

// The multi-block exact sort of one long run [s, s + L) of (keys, vals),
// through (tk, tv)[s, s + L) as the second buffer.
static int merge_sort_run(Ctx &c, unsigned long long *keys, int *vals, unsigned long long *tk, int *tv, int *nr,
                          int s, int L, int nT)
{
    unsigned long long *sk = keys + s, *dk = tk + s;
    int *sv = vals + s, *dv = tv + s;
    const long long threads = ((long long)L + kMergeChunk - 1) / kMergeChunk;
    const unsigned blocks = (unsigned)((threads + 255) / 256);
    for (long long w = 1; w < L; w <<= 1) {
        k_merge_level<<<blocks, 256, 0, c.stream>>>(sk, sv, dk, dv, L, (int)w, alpha_geom_tris(c), c.edges, c.opos,
                                                     nT, c.ctr);
        count_launch();
        std::swap(sk, dk);
        std::swap(sv, dv);
    }
    GALPHA_CUDA(cudaGetLastError());
    if (sk != keys + s) {
        launch_n(c, CopyElems<unsigned long long>{keys + s, sk}, L);
        launch_n(c, CopyElems<int>{vals + s, sv}, L);
    }
    launch_n(c, RunFlags{vals, nr, alpha_geom_tris(c), c.edges, c.opos, s, nT, c.ctr}, L - 1);
    return GPUDT_OK;
}

struct ScatterRanks {
    const unsigned long long *keys;
    const int *vals, *nr, *excl;
    int *tri_ro, *edge_ro;
    double *spectrum;
    int nT;
    const Counters *ct;
    __device__ void operator()(long long ii) const
    {
        if (ct->err) return;  // as in ExactAdjacent
        int i = (int)ii;
        int r = excl[i] + nr[i];
        if (i == 0) {
            spectrum[0] = 0.0;
            return;
        }
        int v = vals[i];
        if (v < nT) tri_ro[v] = r;
        else edge_ro[v - nT] = r;
        if (nr[i]) spectrum[r] = __longlong_as_double((long long)keys[i]);
    }
};

// Intervals of the edges a triangle owns and, from them, of its vertices: the
// triangle's contributions to a vertex are combined before the atomics (1.5
// owned edges on average reach 2.5 vertices, not 3), and the triangles are
// read in order, where one thread per edge gathered a 16-byte record and a
// link each.  The intervals start as all ones: -1 for the signed maximum, the
// largest value for the unsigned minimum, and (-1, -1) for a vertex without
// edges, so no launch sets them up or converts them.
struct EdgeIntervals {
    const int4 *cv, *cn;
    const int *e_off, *tri_ro, *edge_ro;
    int2 *edge_nu;
    int2 *pt;
    __device__ __forceinline__ void global(int v, int lo, int hi) const
    {
        atomicMin((unsigned *)&pt[v].x, (unsigned)lo);
        atomicMax(&pt[v].y, hi);
    }
    // the edges of triangle t; put(vertex, smallest rank, largest rank)
    template <class Put>
    __device__ __forceinline__ void edges(long long t, Put put) const
    {
        const int4 v = cv[t], n = cn[t];
        const int tr = tri_ro[t];
        int e = e_off[t];
        int o[3], lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {-1, -1, -1};
        bool own[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const int nb = geti(n, i);
            own[i] = geti(v, p1(i)) < geti(v, m1(i)) || nb == -1;
            o[i] = own[i] && nb != -1 ? tri_ro[dtri(nb)] : 0;
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
            if (!own[i]) continue;
            int2 nu;
            if (geti(n, i) == -1) nu = make_int2(tr, 0);
            else nu = tr <= o[i] ? make_int2(tr, o[i]) : make_int2(o[i], tr);
            edge_nu[e] = nu;
            const int ro = edge_ro[e];
            const int vmin = ro != 0 ? ro : nu.x;
            e++;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                if (q == i) continue;
                lo[q] = min(lo[q], vmin);
                hi[q] = max(hi[q], nu.y);
            }
        }
#pragma unroll
        for (int q = 0; q < 3; q++)
            if (hi[q] >= 0) put(geti(v, q), lo[q], hi[q]);
    }
    __device__ void operator()(long long t) const
    {
        edges(t, [this](int v, int lo, int hi) { global(v, lo, hi); });
    }
};

// The same with a block's contributions combined in shared memory first: the
// atomics on the vertices bound the plain form (8.0 M triangles: 343 us, 40 M
// atomics), and 1,024 consecutive triangles, which lie together, reach some 650
// vertices 2,560 times.  A vertex that finds no slot of the table in kEiProbes
// steps goes to global memory at once.  231 us at 8.0 M triangles.  Below kEiMany
// triangles per SM (606,208 on 148), fewer tiles than four each, the plain form:
// its threads all start at once there and the atomics no longer bound it
// (100,000 triangles: 6 us).
constexpr int kEiThreads = 256, kEiItems = 4, kEiSlots = 2048, kEiProbes = 4;
constexpr int kEiMany = 4 * kEiThreads * kEiItems;  // triangles per SM

__global__ void __launch_bounds__(kEiThreads) k_edge_intervals(EdgeIntervals f, int nT)
{
    __shared__ int key[kEiSlots], hi_[kEiSlots];
    __shared__ unsigned lo_[kEiSlots];
    for (int i = threadIdx.x; i < kEiSlots; i += kEiThreads) {
        key[i] = -1;
        lo_[i] = 0xffffffffu;
        hi_[i] = -1;
    }
    __syncthreads();
    const long long t0 = (long long)blockIdx.x * (kEiThreads * kEiItems) + threadIdx.x;
#pragma unroll 1
    for (int u = 0; u < kEiItems; u++) {
        const long long t = t0 + u * kEiThreads;
        if (t >= nT) break;
        f.edges(t, [&](int v, int lo, int hi) {
            unsigned s = (unsigned)v * 0x9e3779b1u >> 21;
            for (int k = 0; k < kEiProbes; k++, s = (s + 1) & (kEiSlots - 1)) {
                int was = *(volatile int *)&key[s];
                if (was == -1) was = atomicCAS(&key[s], -1, v);
                if (was == -1 || was == v) {
                    atomicMin(&lo_[s], (unsigned)lo);
                    atomicMax(&hi_[s], hi);
                    return;
                }
            }
            f.global(v, lo, hi);
        });
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kEiSlots; i += kEiThreads)
        if (key[i] >= 0) f.global(key[i], (int)lo_[i], hi_[i]);
}

static void launch_edge_intervals(Ctx &c, const EdgeIntervals &f, int nT)
{
    if (nT < kEiMany * c.sm_count) {
        launch_n(c, f, nT);
        return;
    }
    constexpr int tile = kEiThreads * kEiItems;
    k_edge_intervals<<<(nT + tile - 1) / tile, kEiThreads, 0, c.stream>>>(f, nT);
    count_launch();
}

// ------------------------------------------------------- batched segments
// Set of each value-sorted entry (triangle, or the triangle that owns the edge).
// Set of every entry id in entry order (triangles, then edges in triangle
// order): coalesced reads, so the sorted entries need one gather each.
// First edge of each set (and [K] = nE): edges are numbered in triangle
// order and triangles are grouped by set.
struct SetEdgeBases {
    const int *e_off, *tbase;
    int nT, nE;
    int *ebase;
    __device__ void operator()(long long s) const
    {
        const int t = tbase[s];
        ebase[s] = t < nT ? e_off[t] : nE;
    }
};

// Set of each value-sorted entry, by binary search of its id in the per-set
// bases (triangles and edges are each grouped by set, bases non-decreasing;
// the last set whose base is at most the id owns it) -- no gather by id.
// A coarse table gives the owner of every kEntryBlock-th id, so the search
// runs only over the sets that start inside the entry's block.
constexpr int kEntryBlockBits = 10;

__device__ __forceinline__ int set_owner(const int *b, int lo, int hi, int x)
{
    // the answer lies in [lo, hi): b[lo] <= x < b[hi]
    while (hi - lo > 1) {
        const int m = (lo + hi) >> 1;
        if (b[m] <= x) lo = m;
        else hi = m;
    }
    return lo;
}

// coarse[j]: owner of id j << kEntryBlockBits, for the triangle ids (j <
// nbt) and then the edge ids
struct EntryBlocks {
    const int *tbase, *ebase;
    int K, nbt;
    int *coarse;
    __device__ void operator()(long long jj) const
    {
        const int j = (int)jj;
        const bool tri = j < nbt;
        const int x = (tri ? j : j - nbt) << kEntryBlockBits;
        coarse[j] = set_owner(tri ? tbase : ebase, 0, K, x);
    }
};

struct EntrySet {
    const int *vals;
    const int *tbase, *ebase;
    const int *coarse;
    int K, nT, nbt, nbe;
    unsigned *key;
    __device__ void operator()(long long i) const
    {
        const int v = vals[i];
        const bool tri = v < nT;
        const int *b = tri ? tbase : ebase;
        const int x = tri ? v : v - nT;
        const int j = x >> kEntryBlockBits;
        const int *cb = tri ? coarse : coarse + nbt;
        const int nb = tri ? nbt : nbe;
        // the owner of the block's first id, up to the owner of the next block's
        const int lo = cb[j], hi = j + 1 < nb ? min(K, cb[j + 1] + 1) : K;
        key[i] = (unsigned)set_owner(b, lo, hi, x);
    }
};

struct SetOfSorted {
    const unsigned *setkey;
    int *seg;  // indexed like the full entry array (entry 0 = sentinel)
    __device__ void operator()(long long i) const
    {
        seg[1 + i] = (int)setkey[i];
        if (i == 0) seg[0] = -1;
    }
};

// Per set: the global rank count before its first entry, and its number of
// distinct values (entries of a set are contiguous; each set's first entry
// starts a rank).
struct SetRankBounds {
    const int *seg, *nr, *excl;
    int n;
    int *firstexcl, *endrank;
    __device__ void operator()(long long ii) const
    {
        int i = (int)ii;
        if (i == 0) return;
        int s = seg[i];
        if (i == 1 || seg[i - 1] != s) firstexcl[s] = excl[i];
        if (i == n - 1 || seg[i + 1] != s) endrank[s] = excl[i] + nr[i];
    }
};

struct SetDistinct {
    const int *firstexcl;
    int *nd;  // in: end rank (0 for a set without entries); out: distinct values
    __device__ void operator()(long long s) const { nd[s] -= firstexcl[s]; }
};

struct ScatterRanksSeg {
    const unsigned long long *keys;
    const int *vals, *nr, *excl, *seg, *firstexcl, *spec_off;
    int *tri_ro, *edge_ro;
    double *spectrum;
    int nT;
    __device__ void operator()(long long ii) const
    {
        int i = (int)ii;
        if (i == 0) return;
        int s = seg[i];
        int r = excl[i] + nr[i] - firstexcl[s];
        int v = vals[i];
        if (v < nT) tri_ro[v] = r;
        else edge_ro[v - nT] = r;
        if (nr[i]) spectrum[spec_off[s] + s + r] = __longlong_as_double((long long)keys[i]);
    }
};

struct SetSentinels {
    const int *spec_off;
    double *spectrum;
    __device__ void operator()(long long s) const { spectrum[spec_off[s] + s] = 0.0; }
};

// ------------------------------------------------------------------ stage
// Up to this many entries the host looks at nothing between the sort and the
// intervals: what it would have looked for (a long group of equal key tops, a
// run out of exact order) then costs a second pass over the ranks, about 40 us
// at this size, where the two reads cost 30 us on every call.
constexpr int kDeferEntries = 1 << 19;

// Ranks of the sorted entries (keys, vals): near-equal neighbours compared
// exactly, runs out of exact order re-sorted.  With `defer` such runs are only
// counted (al_slow) and the host reads nothing.
static int alpha_ranks(Ctx &c, AlphaSegs *segs, int nIn, bool defer)
{
    int r;
    const int nT = c.nT_out;
    const int *seg = segs ? segs->seg : nullptr;
    int *nr = c.aux, *unc = c.list, *slow = c.list2, *slowflag = c.stamp;
    launch_n(c, MarkRuns{c.keys, nr, unc, nIn, c.ctr, seg}, nIn);
    const ExactAdjacent adj{c.keys, c.vals, nr, slow, defer ? nullptr : slowflag, unc, alpha_geom_tris(c), c.edges,
                            c.opos, nT, c.ctr, seg};
    if (defer) {
        launch_dev(c, adj, &c.ctr->al_unc, nIn);
        return GPUDT_OK;
    }
    r = read_counters(c);
    if (r) return r;
    if (c.hctr->al_unc == 0) return GPUDT_OK;
    GALPHA_CUDA(cudaMemsetAsync(slowflag, 0, sizeof(int) * (size_t)nIn, c.stream));
    launch_n(c, adj, c.hctr->al_unc);
    r = read_counters(c);
    if (r) return r;
    if (c.hctr->err) return stage_fail(c, c.hctr->err, "alpha");
    if (c.hctr->al_slow == 0) return GPUDT_OK;
    // runs longer than kThreadRun are listed after the slow runs
    const int nslow = c.hctr->al_slow;
    int *longs = slow + nslow;
    GALPHA_CUDA(cudaMemsetAsync(&c.ctr->nlong, 0, sizeof(int), c.stream));
    launch_n(c, ResolveRuns{c.keys, c.vals, nr, slow, alpha_geom_tris(c), c.edges, c.opos, nIn, nT, c.ctr, seg, longs},
             nslow);
    r = read_counters(c);
    if (r) return r;
    if (c.hctr->err) return stage_fail(c, c.hctr->err, "alpha");
    if (c.hctr->nlong == 0) return GPUDT_OK;
    // (keys2, vals2) are free now: the second buffer of each run's merge sort
    const int nlong = c.hctr->nlong;
    // runs for the multi-block merge: (start, length) pairs after the long runs, 8-byte aligned
    uintptr_t hp = reinterpret_cast<uintptr_t>(longs + nlong);
    int2 *huge = reinterpret_cast<int2 *>((hp + 7) & ~(uintptr_t)7);
    GALPHA_CUDA(cudaMemsetAsync(&c.ctr->nhuge, 0, sizeof(int), c.stream));
    k_resolve_long<<<(unsigned)nlong, kLongThreads, 0, c.stream>>>(c.keys, c.vals, nr, c.keys2, c.vals2, longs,
                                                                   alpha_geom_tris(c), c.edges, c.opos, nIn, nT, c.ctr,
                                                                   seg, c.block_run, huge);
    count_launch();
    GALPHA_CUDA(cudaGetLastError());
    r = read_counters(c);
    if (r) return r;
    if (c.hctr->err) return stage_fail(c, c.hctr->err, "alpha");
    const int nhuge = c.hctr->nhuge;
    if (nhuge > 0) {
        std::vector<int2> hs(nhuge);
        r = read_small(c, hs.data(), huge, sizeof(int2) * (size_t)nhuge);
        if (r) return r;
        for (const int2 &h : hs) {
            r = merge_sort_run(c, c.keys, c.vals, c.keys2, c.vals2, nr, h.x, h.y, nT);
            if (r) return r;
        }
        r = read_counters(c);
        if (r) return r;
        if (c.hctr->err) return stage_fail(c, c.hctr->err, "alpha");
    }
    return GPUDT_OK;
}

// Intervals of edges and vertices; again: not for the first time since the
// keys, which start the vertex intervals.
static int alpha_intervals(Ctx &c, bool again)
{
    const int nT = c.nT_out;
    if (again) GALPHA_CUDA(cudaMemsetAsync(c.pt_nu, 0xff, sizeof(int2) * (size_t)c.N, c.stream));
    launch_edge_intervals(c, EdgeIntervals{c.cv, c.cn, c.e_off, c.tri_ro, c.edge_ro, c.edge_nu, c.pt_nu}, nT);
    GALPHA_CUDA(cudaGetLastError());
    return read_counters(c);
}

// Up to kBlockSort entries: the sort, the ranks and the spectrum in one launch
// of one block, the sorted entries kept in shared memory between them; neighbours
// within 2 ulp are compared exactly on the spot, and a run out of exact order
// is only counted (al_slow): the caller then redoes the ranks from the sorted
// entries, which are written back.  (nT and the number of unattached edges are
// on the device, so the host need not look before the launch.)  The usual
// five digits of the key tops come first; only when they leave equal tops out
// of order (the block knows) are all eight sorted.  1,000 points (3,905 entries):
// 34 us, 2,000 points (7,888): 54, where the passes, the group fix-up, the flags,
// the scan and the scatter were 13 launches and 85 us, and a counter read.
__global__ void __launch_bounds__(kBsThreads) k_alpha_rank_block(unsigned long long *keys, int *vals, int nT,
                                                                 const int4 *cv, const int *edges, const double2 *P,
                                                                 int *tri_ro, int *edge_ro, double *spectrum,
                                                                 Counters *ct)
{
    extern __shared__ __align__(16) unsigned char bs_smem[];
    typedef unsigned long long K;
    BsSmem<K> &S = *reinterpret_cast<BsSmem<K> *>(bs_smem);
    __shared__ int s_warp[kBsWarps];
    const int n = nT + ct->al_unatt;
    if (n > kBlockSort || ct->err) return;
    auto load = [&](int i, K &k, int &v) {
        k = keys[1 + i];
        v = vals[1 + i];
    };
    auto store = [&](int i, K k, int v) {
        keys[1 + i] = k;
        vals[1 + i] = v;
    };
    block_sort(S, n, 24, 5, load, store);
    bool off = false;  // a pair with equal tops in the wrong order
    for (int i = 1 + threadIdx.x; i < n; i += kBsThreads) off |= S.key[i] < S.key[i - 1];
    if (__syncthreads_or(off)) {  // stable: from the top's order as from any other
        block_sort(S, n, 0, 8, load, store);
        if (threadIdx.x == 0) ct->fx_many = 1;
        __syncthreads();
    }
    // S.key / S.val hold the sorted entries; the warp's entries in order, 32 at a time
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int rounds = (n + kBsThreads - 1) / kBsThreads, base = w * rounds * 32;
    unsigned starts[kBlockSort / kBsThreads];
    int before = 0;
#pragma unroll
    for (int r = 0; r < kBlockSort / kBsThreads; r++) {
        if (r >= rounds) break;
        const int i = base + r * 32 + lane;
        bool st = i < n;
        if (st && i > 0 && near_equal(S.key[i - 1], S.key[i])) {
            const int cmp = exact_cmp_vals(S.val[i - 1], S.val[i], nT, cv, edges, P);
            atomicAdd(&ct->exact_compares, 1ull);
            if (cmp == EXACT_OVERFLOW) set_err(ct, GPUDT_ERR_EXACT, 110);
            else if (cmp == 0) {
                st = false;
                atomicAdd(&ct->nties, 1);
            } else if (cmp > 0) atomicAdd(&ct->al_slow, 1);
        }
        starts[r] = __ballot_sync(0xffffffffu, st);
        before += __popc(starts[r]);
    }
    if (lane == 0) s_warp[w] = before;
    __syncthreads();
    int rank = 0, total = 0;
    for (int q = 0; q < kBsWarps; q++) {
        const int x = s_warp[q];
        if (q < w) rank += x;
        total += x;
    }
#pragma unroll
    for (int r = 0; r < kBlockSort / kBsThreads; r++) {
        if (r >= rounds) break;
        const int i = base + r * 32 + lane;
        if (i < n) {
            const int k = rank + __popc(starts[r] & (0xffffffffu >> (31 - lane)));  // starts up to this entry
            const int v = S.val[i];
            if (v < nT) tri_ro[v] = k;
            else edge_ro[v - nT] = k;
            if ((starts[r] >> lane) & 1u) spectrum[k] = __longlong_as_double((long long)S.key[i]);
        }
        rank += __popc(starts[r]);
    }
    if (threadIdx.x == 0) {
        spectrum[0] = 0.0;
        ct->al_ranks = total;
    }
}

// Spectrum, simplex ranks and intervals from the rank-start flags (c.aux).
static int alpha_scatter(Ctx &c, AlphaSegs *segs, int nIn, bool again = false)
{
    const int nT = c.nT_out;
    const int *nr = c.aux;
    int r = exclusive_scan_int(c, nr, c.rank, nIn, &c.ctr->al_ranks);
    if (r) return r;
    if (!segs) {
        launch_n(c, ScatterRanks{c.keys, c.vals, nr, c.rank, c.tri_ro, c.edge_ro, c.spectrum, nT, c.ctr}, nIn);
    } else {
        GALPHA_CUDA(cudaMemsetAsync(segs->nd, 0, sizeof(int) * (size_t)segs->K, c.stream));
        GALPHA_CUDA(cudaMemsetAsync(segs->firstexcl, 0, sizeof(int) * (size_t)segs->K, c.stream));
        launch_n(c, SetRankBounds{segs->seg, nr, c.rank, nIn, segs->firstexcl, segs->nd}, nIn);
        launch_n(c, SetDistinct{segs->firstexcl, segs->nd}, segs->K);
        r = exclusive_scan_int(c, segs->nd, segs->spec_off, segs->K, nullptr);
        if (r) return r;
        launch_n(c, ScatterRanksSeg{c.keys, c.vals, nr, c.rank, segs->seg, segs->firstexcl, segs->spec_off,
                                    c.tri_ro, c.edge_ro, c.spectrum, nT},
                 nIn);
        launch_n(c, SetSentinels{segs->spec_off, c.spectrum}, segs->K);
    }
    return alpha_intervals(c, again);
}

int stage_alpha(Ctx &c, AlphaSegs *segs)
{
    int r;
    const int nT = c.nT_out;
    // an alpha call on a resident mesh starts without the error of an earlier
    // failed alpha call and with its own counts
    GALPHA_CUDA(cudaMemsetAsync(&c.ctr->err, 0, kAlphaBytes, c.stream));
    const bool few = nT <= kAkFew * c.sm_count;
    const int tile = kAkThreads * (few ? 1 : kAkItemsMany), tiles = (nT + tile - 1) / tile;
    if (nT > 0) {
        // status words in the counter block, or in the sort's scratch, which no sort uses yet
        unsigned long long *status = c.ctr->al_status;
        if (tiles + 1 > 64) {
            status = (unsigned long long *)c.rhist;
            GALPHA_CUDA(cudaMemsetAsync(status, 0, sizeof(unsigned long long) * (size_t)(tiles + 1), c.stream));
        }
        const AlphaKeysArgs a{c.cv, c.cn, alpha_geom_tris(c), c.opos, nT, c.e_off, c.keys, c.vals, c.edges, c.edge_ro,
                              c.list, status, tiles, c.pt_nu, c.N, c.ctr};
        if (few) k_alpha_keys<1><<<(unsigned)tiles, kAkThreads, 0, c.stream>>>(a);
        else k_alpha_keys<kAkItemsMany><<<(unsigned)tiles, kAkThreads, 0, c.stream>>>(a);
        count_launch();
    } else if (c.N > 0) {
        GALPHA_CUDA(cudaMemsetAsync(c.pt_nu, 0xff, sizeof(int2) * (size_t)c.N, c.stream));
    }
    // the sliver list's length stays on the device
    launch_dev(c, SliverKeys{alpha_geom_tris(c), c.opos, c.list, c.keys, c.ctr}, &c.ctr->al_sliver, nT);
    auto sort_begins = [&]() {
        c.sort_passes = 0;
        if (c.events) {
            cudaEventRecord(c.kev[8], c.stream);
            c.kev_rec[8] = true;
        }
    };
    auto sort_ends = [&]() {
        if (c.events) {
            cudaEventRecord(c.kev[9], c.stream);
            c.kev_rec[9] = true;
        }
    };
    auto rank_block = [&]() {
        static bool set[64];
        const int smem = (int)sizeof(BsSmem<unsigned long long>);
        int e = block_sort_attr(c, k_alpha_rank_block, smem, set);
        if (e) return e;
        sort_begins();
        c.sort_passes = 5;
        k_alpha_rank_block<<<1, kBsThreads, smem, c.stream>>>(c.keys, c.vals, nT, alpha_geom_tris(c), c.edges, c.opos,
                                                              c.tri_ro, c.edge_ro, c.spectrum, c.ctr);
        count_launch();
        sort_ends();
        return alpha_intervals(c, false);
    };
    // a triangle owns at most three edges: this few cannot pass kBlockSort entries
    const bool blind = !segs && 4ll * nT <= kBlockSort;
    r = blind ? rank_block() : read_counters(c);
    if (r) return r;
    if (c.hctr->err) return stage_fail(c, c.hctr->err, "alpha");
    const int nE = c.hctr->al_edges;
    c.nE = nE;
    const int nIn = 1 + nT + c.hctr->al_unatt;
    c.nSpecIn = nIn;
    if (!segs && nIn - 1 <= kBlockSort) {
        if (!blind) r = rank_block();
        if (r) return r;
        c.st.sortKeys = nIn - 1;
        if (c.hctr->fx_many) c.sort_passes += 8;
        c.st.sortPasses = c.sort_passes;
        if (!c.hctr->err && c.hctr->al_slow) {  // a run out of exact order: the ranks again
            GALPHA_CUDA(cudaMemsetAsync(&c.ctr->fx_groups, 0, kRankBytes, c.stream));
            r = alpha_ranks(c, segs, nIn, false);
            if (!r) r = alpha_scatter(c, segs, nIn, true);
            if (r) return r;
        }
        if (c.hctr->err) return stage_fail(c, c.hctr->err, "alpha");
        c.nSpec = c.hctr->al_ranks + 1;
        return GPUDT_OK;
    }
    sort_begins();
    bool second = false;
    // entry 0 is the sentinel (no key of its own); a batch's entries are
    // regrouped after the sort, so a late look at its long groups is no option
    const bool defer = !segs && nIn <= kDeferEntries;
    unsigned long long *k1 = c.keys, *k2 = c.keys2;
    int *v1 = c.vals, *v2 = c.vals2;
    r = radix_sort(c, k1 + 1, v1 + 1, k2 + 1, v2 + 1, nIn - 1, &second, defer);
    if (r) return r;
    // the sorted entries may be in the second buffers: they become keys / vals
    // for the rest of this result's life
    auto take_sorted = [&]() {
        c.keys = second ? k2 : k1;
        c.keys2 = second ? k1 : k2;
        c.vals = second ? v2 : v1;
        c.vals2 = second ? v1 : v2;
    };
    take_sorted();
    sort_ends();
    c.st.sortKeys = nIn - 1;
    c.st.sortPasses = c.sort_passes;
    if (segs) {
        // stable sort by set, carrying each entry's key and value: entries end
        // up ordered by (set, value)
        const int m = nIn - 1;
        unsigned *ka = (unsigned *)c.rank, *kb = (unsigned *)c.aux2;  // both free until the ranks
        launch_n(c, SetEdgeBases{c.e_off, segs->tbase, nT, nE, segs->ebase}, segs->K + 1);
        // c.list is free here (the sliver list has been consumed)
        const int nbt = (nT >> kEntryBlockBits) + 1, nbe = (nE >> kEntryBlockBits) + 1;
        int *coarse = c.list;
        launch_n(c, EntryBlocks{segs->tbase, segs->ebase, segs->K, nbt, coarse}, nbt + nbe);
        launch_n(c, EntrySet{c.vals + 1, segs->tbase, segs->ebase, coarse, segs->K, nT, nbt, nbe, ka}, m);
        int bits = 0;
        while ((1ll << bits) < segs->K) bits++;
        r = radix_sort_set_kv(c, ka, kb, c.keys + 1, c.vals + 1, c.keys2 + 1, c.vals2 + 1, m, bits);
        if (r) return r;
        launch_n(c, SetOfSorted{ka, segs->seg}, m);
    }
    r = alpha_ranks(c, segs, nIn, defer);
    if (!r) r = alpha_scatter(c, segs, nIn);
    if (r) return r;
    if (c.hctr->err) return stage_fail(c, c.hctr->err, "alpha");
    if (defer && (c.hctr->fx_long || c.hctr->fx_many || c.hctr->al_slow)) {
        // a long group or a run out of order after all: that, and the ranks again
        if (c.hctr->fx_long || c.hctr->fx_many) {
            r = radix_sort_finish(c, k1 + 1, v1 + 1, k2 + 1, v2 + 1, nIn - 1, &second, false);
            if (r) return r;
            take_sorted();
            c.st.sortPasses = c.sort_passes;
        }
        GALPHA_CUDA(cudaMemsetAsync(&c.ctr->fx_groups, 0, kRankBytes, c.stream));
        r = alpha_ranks(c, segs, nIn, false);
        if (!r) r = alpha_scatter(c, segs, nIn, true);
        if (r) return r;
        if (c.hctr->err) return stage_fail(c, c.hctr->err, "alpha");
    }
    c.nSpec = c.hctr->al_ranks + (segs ? segs->K : 1);  // distinct ranks incl. the sentinel(s)
    return GPUDT_OK;
}

// ------------------------------------------------------------ alpha query
// Classification of every simplex of the alpha complex at a value alpha
// (a squared radius, the unit of the spectrum), from the intervals above:
// R = the largest rank with spectrum[R] <= alpha, then
//   triangle:  ro <= R                                    -> interior
//   edge:      nu_max != 0 (finite) && nu_max <= R        -> interior
//              nu_min <= R                                -> regular
//              ro != 0 (unattached) && ro <= R            -> singular
//   point:     (nu_min, nu_max) the same way, with the singular interval
//              starting at rank 0 (every vertex is in the complex at alpha >= 0)
//   otherwise exterior.  Points dropped as duplicates (no incident edge) are
// exterior.  These are the interval semantics of kernel.cu:427-624 that the
// reference's viewer draws from (Visualizer.cu:296-337: an edge is drawn from
// its ro / nu_min entry until its nu_max entry, a triangle from its ro entry).
namespace {

__device__ __forceinline__ int interval_class(int ro, int nu_min, int nu_max, int R)
{
    if (nu_max > 0 && nu_max <= R) return 3;
    if (nu_min <= R) return 2;
    if (ro >= 0 && ro <= R) return 1;
    return 0;
}

// Largest index r in [lo, n) with sp[r] <= a, given sp[lo] <= a (one whole
// warp; every lane gets r).  The 32 entries after lo are tried first: a
// quantile's value is its own answer unless neighbours round to the same
// double, and then each step splits the rest in 33.
template <class T>
__device__ __forceinline__ int warp_last_leq(const T *__restrict__ sp, int lo, int n, T a)
{
    const int lane = threadIdx.x & 31;
    int hi = n - 1;  // the answer lies in [lo, hi]
    for (bool near = true; lo < hi; near = false) {
        const int step = near ? 1 : (hi - lo + 32) / 33;
        const int i = (int)min((long long)hi, (long long)lo + (long long)(lane + 1) * step);
        const unsigned m = __ballot_sync(0xffffffffu, sp[i] <= a);  // a prefix of the lanes
        const int k = __popc(m);
        const int base = lo;
        lo = (int)min((long long)hi, (long long)base + (long long)k * step);
        if (k < 32) hi = (int)min((long long)hi, max((long long)lo, (long long)base + (long long)(k + 1) * step - 1));
    }
    return lo;
}

// Rank of a query: the value (given, or the spectrum's at a quantile) and the
// largest rank whose spectrum value is at most it, -1 for a negative value.
__device__ __forceinline__ int warp_query_rank(const double *__restrict__ sp, int n, double q, int by_quantile,
                                               double *alpha)
{
    double a = q;
    int lo = 0;  // spectrum[0] = 0
    if (by_quantile) {
        const double qq = q < 0.0 ? 0.0 : (q > 1.0 ? 1.0 : q);
        lo = (int)llrint(qq * (double)(n - 1));
        a = sp[lo];
    }
    *alpha = a;
    return a >= 0.0 ? warp_last_leq(sp, lo, n, a) : -1;
}

// The classified arrays: points, then edges, then triangles.  A block takes
// chunks of kQChunk consecutive entries of one kind.  The kernel reads 8, 12
// and 4 bytes and writes one byte per entry, so it is bound by memory as long
// as its counts stay in registers: with one atomic per warp on the twelve
// shared counters a query took 860 us at 4.2 M points, 23 times the 37 us that
// its 243 MB take at the copy rate; with register counts it takes 58 us.
struct QueryArrays {
    const int2 *__restrict__ pt;
    const int *__restrict__ edge_ro;
    const int2 *__restrict__ edge_nu;
    const int *__restrict__ tri_ro;
    uint8_t *__restrict__ cls;
    int N, nE, nT;
};

constexpr int kQThreads = 256, kQItems = 8, kQChunk = kQThreads * kQItems;

__host__ __device__ inline int q_chunks(int n) { return n / kQChunk + (n % kQChunk != 0); }

// This thread's entries e0 + u * kQThreads < n of one kind (0 points, 1 edges,
// 2 triangles): load() puts all loads in flight; classify() stores their
// classes at the ranks rank(u) and hands them to count(u, class).
struct QChunk {
    int ro[kQItems];
    int2 nu[kQItems];
    __device__ __forceinline__ void load(const QueryArrays &A, int kind, int e0, int n)
    {
#pragma unroll
        for (int u = 0; u < kQItems; u++) {
            const int e = e0 + u * kQThreads;
            if (e >= n) continue;
            if (kind == 0) nu[u] = A.pt[e];
            else if (kind == 1) {
                ro[u] = A.edge_ro[e];
                nu[u] = A.edge_nu[e];
            } else ro[u] = A.tri_ro[e];
        }
    }
    template <class Rank, class Count>
    __device__ __forceinline__ void classify(const QueryArrays &A, int kind, int e0, int n, Rank rank, Count count) const
    {
        uint8_t *out = A.cls + (kind == 0 ? 0ll : kind == 1 ? (long long)A.N : (long long)A.N + A.nE);
#pragma unroll
        for (int u = 0; u < kQItems; u++) {
            const int e = e0 + u * kQThreads;
            if (e >= n) continue;
            const int R = rank(u);
            int k;
            if (kind == 0) k = (nu[u].x < 0 || R < 0) ? 0 : interval_class(0, nu[u].x, nu[u].y, R);
            else if (kind == 1) k = R < 0 ? 0 : interval_class(ro[u] != 0 ? ro[u] : -1, nu[u].x, nu[u].y, R);
            else k = (R >= 0 && ro[u] <= R) ? 3 : 0;
            out[e] = (uint8_t)k;
            count(u, k);
        }
    }
};

// Four class counts of up to 65,535 each in one word.
__device__ __forceinline__ unsigned long long warp_sum64(unsigned long long v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One query of a single set: every block finds the rank itself (two loads in
// a row for a quantile), so the query is one launch; the last block to finish
// hands the counts to the host's mirror and clears them for the next query.
__global__ void __launch_bounds__(kQThreads) k_query(QueryArrays A, const double *__restrict__ spectrum, int nSpec,
                                                     double q, int by_quantile, Counters *ct, Counters *host)
{
    __shared__ int s_R, s_cnt[12], s_last;
    if (threadIdx.x < 12) s_cnt[threadIdx.x] = 0;
    if (threadIdx.x < 32) {
        double a;
        const int R = warp_query_rank(spectrum, nSpec, q, by_quantile, &a);
        if (threadIdx.x == 0) {
            s_R = R;
            if (blockIdx.x == 0) {
                ct->qrank = R;
                ct->qalpha = a;
            }
        }
    }
    __syncthreads();
    const int R = s_R;
    const int cp = q_chunks(A.N), ce = q_chunks(A.nE), chunks = cp + ce + q_chunks(A.nT);
    // class counts, 16 bits each: at most 6 * 2^28 entries in chunks of 8 per
    // thread over 8 blocks per SM are under 6,000 per thread
    unsigned long long acc[3] = {0ull, 0ull, 0ull};
    for (int ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
        const int kind = ch < cp ? 0 : (ch < cp + ce ? 1 : 2);
        const int c0 = ch - (kind == 0 ? 0 : kind == 1 ? cp : cp + ce);
        unsigned long long n = 0ull;
        // c0 * kQChunk < 2^31 - kQChunk (entry counts stay below 1.7e9), so e0 + 7 * 256 does not wrap
        const int e0 = c0 * kQChunk + (int)threadIdx.x, ne = kind == 0 ? A.N : kind == 1 ? A.nE : A.nT;
        QChunk Q;
        Q.load(A, kind, e0, ne);
        Q.classify(A, kind, e0, ne, [&](int) { return R; }, [&](int, int k) { n += 1ull << (16 * k); });
        if (kind == 0) acc[0] += n;
        else if (kind == 1) acc[1] += n;
        else acc[2] += n;
    }
#pragma unroll
    for (int kind = 0; kind < 3; kind++) {
        unsigned v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = __reduce_add_sync(0xffffffffu, (unsigned)(acc[kind] >> (16 * k)) & 0xffffu);
        const int k = threadIdx.x & 31;
        const unsigned x = k == 0 ? v[0] : k == 1 ? v[1] : k == 2 ? v[2] : v[3];
        if (k < 4 && x) atomicAdd(&s_cnt[kind * 4 + k], (int)x);
    }
    __syncthreads();
    if (threadIdx.x < 12 && s_cnt[threadIdx.x]) atomicAdd(&ct->qcount[threadIdx.x], s_cnt[threadIdx.x]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&ct->qdone, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x < 12) {
        host->qcount[threadIdx.x] = *(volatile int *)&ct->qcount[threadIdx.x];
        ct->qcount[threadIdx.x] = 0;
    } else if (threadIdx.x == 12) {
        host->qrank = *(volatile int *)&ct->qrank;
        host->qalpha = *(volatile double *)&ct->qalpha;
        host->err = ct->err;
        ct->qdone = 0;
    }
    __threadfence_system();
}

// Per set of a batch (one warp each): the set's spectrum is
// spectrum[spec_off[s] + s ..] of length nd[s] + 1 (its own rank-0 sentinel
// first).
__global__ void __launch_bounds__(kQThreads) k_query_ranks(const double *__restrict__ spectrum,
                                                           const int *__restrict__ spec_off,
                                                           const int *__restrict__ nd,
                                                           const double *__restrict__ param, int by_quantile, int K,
                                                           int *R, double *alpha, int *counts)
{
    const int s = blockIdx.x * (kQThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (s >= K) return;
    double a;
    const int r = warp_query_rank(spectrum + spec_off[s] + s, nd[s] + 1, param[s], by_quantile, &a);
    if (lane == 0) {
        R[s] = r;
        alpha[s] = a;
    }
    if (lane < 12) counts[12 * (long long)s + lane] = 0;
}

// Last set in [lo, hi] whose base is at most x, base[lo] <= x.
__device__ __forceinline__ int q_set(const int *__restrict__ base, int lo, int hi, int x)
{
    while (lo < hi) {
        const int m = (lo + hi + 1) >> 1;
        if (base[m] <= x) lo = m;
        else hi = m - 1;
    }
    return lo;
}

// A batch's queries.  Points, edges and triangles are grouped by set, so a
// chunk knows its sets from its first and last entry (found by whole warps,
// two rounds of loads for 1,024 sets, behind the chunk's own loads: a binary
// search of ten dependent loads ahead of them kept the kernel at 290 us, it
// now takes 188): a chunk inside one set (most of them)
// counts in registers, one that spans several finds each entry's set between
// those two.  No per-entry set array is read (the edges' sets used to take a
// 16-byte record and a gather each: 296 us per query of 9.7 M points in 1,024
// sets).
__global__ void __launch_bounds__(kQThreads) k_query_sets(QueryArrays A, const int *__restrict__ vbase,
                                                          const int *__restrict__ ebase,
                                                          const int *__restrict__ tbase, int K,
                                                          const int *__restrict__ R, int *counts)
{
    const int cp = q_chunks(A.N), ce = q_chunks(A.nE), chunks = cp + ce + q_chunks(A.nT);
    for (int ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
        const int kind = ch < cp ? 0 : (ch < cp + ce ? 1 : 2);
        const int c0 = (ch - (kind == 0 ? 0 : kind == 1 ? cp : cp + ce)) * kQChunk;
        const int n = kind == 0 ? A.N : kind == 1 ? A.nE : A.nT;
        const int *base = kind == 0 ? vbase : kind == 1 ? ebase : tbase;
        const int e0 = c0 + (int)threadIdx.x;
        QChunk Q;
        Q.load(A, kind, e0, n);
        const int s0 = warp_last_leq(base, 0, K, c0), s1 = warp_last_leq(base, s0, K, min(n - 1, c0 + kQChunk - 1));
        if (s0 == s1) {
            const int r = R[s0];
            unsigned long long acc = 0ull;
            Q.classify(A, kind, e0, n, [&](int) { return r; }, [&](int, int k) { acc += 1ull << (16 * k); });
            acc = warp_sum64(acc);  // at most 256 per class
            const int k = threadIdx.x & 31;
            if (k < 4) {
                const int x = (int)(acc >> (16 * k)) & 0xffff;
                if (x) atomicAdd(&counts[12 * (long long)s0 + kind * 4 + k], x);
            }
        } else {
            int st[kQItems];
#pragma unroll
            for (int u = 0; u < kQItems; u++) {
                const int e = e0 + u * kQThreads;
                st[u] = e < n ? q_set(base, s0, s1, e) : s1;
            }
            Q.classify(A, kind, e0, n, [&](int u) { return R[st[u]]; },
                       [&](int u, int k) {
                           const int bin = st[u] * 12 + kind * 4 + k;
                           const unsigned peers = __match_any_sync(__activemask(), bin);
                           if ((peers & ((1u << (threadIdx.x & 31)) - 1u)) == 0) atomicAdd(&counts[bin], __popc(peers));
                       });
        }
    }
}

QueryArrays query_arrays(const Ctx &c)
{
    return QueryArrays{c.pt_nu, c.edge_ro, c.edge_nu, c.tri_ro, c.qclass, c.N, c.nE, c.nT_out};
}

unsigned query_blocks(const Ctx &c)
{
    const long long chunks = (long long)q_chunks(c.N) + q_chunks(c.nE) + q_chunks(c.nT_out);
    return (unsigned)std::max(1ll, std::min(chunks, (long long)c.sm_count * 8));
}

}  // namespace

int alpha_query_sets(Ctx &c, int K, const int *vbase, const int *ebase, const int *tbase, const int *spec_off,
                     const int *nd, const double *param, int by_quantile, int *R, double *alpha, int *counts)
{
    k_query_ranks<<<(unsigned)((K + kQThreads / 32 - 1) / (kQThreads / 32)), kQThreads, 0, c.stream>>>(
        c.spectrum, spec_off, nd, param, by_quantile, K, R, alpha, counts);
    k_query_sets<<<query_blocks(c), kQThreads, 0, c.stream>>>(query_arrays(c), vbase, ebase, tbase, K, R, counts);
    count_launch(2);
    GALPHA_CUDA(cudaGetLastError());
    return GPUDT_OK;
}

// The query's answer is left in the host mirror's q* fields and err.
int alpha_query(Ctx &c, double alpha, double q, bool by_quantile)
{
    k_query<<<query_blocks(c), kQThreads, 0, c.stream>>>(query_arrays(c), c.spectrum, c.nSpec,
                                                         by_quantile ? q : alpha, by_quantile ? 1 : 0, c.ctr,
                                                         c.hctr_dev);
    count_launch();
    c.host_reads++;
    GALPHA_CUDA(cudaGetLastError());
    GALPHA_CUDA(cudaStreamSynchronize(c.stream));
    return GPUDT_OK;
}

}  // namespace galpha
