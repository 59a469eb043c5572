// block_sort.cuh -- stable radix sort of up to kBlockSort entries by one block.
#pragma once
#include <mutex>
#include "internal.cuh"

namespace galpha {

// Up to kBlockSort entries sorted by one block in one launch: keys and values
// stay in shared memory from the first digit to the last.  A pass of a small
// array by launches of its own is three launches of 2 to 5 us for one tile's
// work, whose latency (ballots, two barriers, one shared-memory round trip) is
// the same here without the launches.  Stable, like the passes: warp w ranks
// its own consecutive entries.
constexpr int kBsThreads = 1024, kBsWarps = kBsThreads / 32;

template <typename K>
struct BsSmem {
    K key[kBlockSort];
    int val[kBlockSort];
    int wcnt[kBsWarps][256];
    int start[256];
    int part[8];
};

// Sorts the n entries (key(i), val(i)) on digits [shift0, shift0 + 8 * passes)
// and hands them out in order.
template <typename K, class Load, class Store>
__device__ __forceinline__ void block_sort(BsSmem<K> &S, int n, int shift0, int passes, Load load, Store store)
{
    constexpr int kMax = kBlockSort / kBsThreads;  // entries per thread at most
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int rounds = (n + kBsThreads - 1) / kBsThreads, per_warp = rounds * 32;
    const unsigned lt = (1u << lane) - 1u;
    K key[kMax];
    int val[kMax], rk[kMax];
#pragma unroll
    for (int r = 0; r < kMax; r++) {
        const int i = w * per_warp + r * 32 + lane;
        if (r < rounds && i < n) load(i, key[r], val[r]);
    }
    for (int p = 0; p < passes; p++) {
        const int shift = shift0 + 8 * p;
        for (int d = lane; d < 256; d += 32) S.wcnt[w][d] = 0;
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kMax; r++) {
            if (r >= rounds) break;
            const bool ok = w * per_warp + r * 32 + lane < n;
            const int dg = (int)((key[r] >> shift) & 255);
            unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const unsigned bb = __ballot_sync(0xffffffffu, (dg >> b) & 1);
                peers &= ((dg >> b) & 1) ? bb : ~bb;
            }
            const int leader = ok ? __ffs(peers) - 1 : lane;
            int before = 0;
            if (ok && lane == leader) before = atomicAdd(&S.wcnt[w][dg], __popc(peers));
            before = __shfl_sync(0xffffffffu, before, leader);
            rk[r] = before + __popc(peers & lt);
        }
        __syncthreads();
        if (threadIdx.x < 256) {  // per digit: warps in order, then the digits in order
            const int d = threadIdx.x;
            int s = 0;
            for (int q = 0; q < kBsWarps; q++) {
                const int c = S.wcnt[q][d];
                S.wcnt[q][d] = s;
                s += c;
            }
            int incl = s;
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) S.part[w] = incl;
            S.start[d] = incl - s;
        }
        __syncthreads();
        if (threadIdx.x < 256) {
            int add = 0;
            for (int q = 0; q < w; q++) add += S.part[q];
            S.start[threadIdx.x] += add;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kMax; r++) {
            const int i = w * per_warp + r * 32 + lane;
            if (r < rounds && i < n) {
                const int dg = (int)((key[r] >> shift) & 255);
                const int at = S.start[dg] + S.wcnt[w][dg] + rk[r];
                S.key[at] = key[r];
                S.val[at] = val[r];
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kMax; r++) {
            const int i = w * per_warp + r * 32 + lane;
            if (r < rounds && i < n) {
                key[r] = S.key[i];
                val[r] = S.val[i];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < kMax; r++) {
        const int i = w * per_warp + r * 32 + lane;
        if (r < rounds && i < n) store(i, key[r], val[r]);
    }
}

// The shared-memory opt-in of a kernel, once per device.
template <class Kernel>
inline int block_sort_attr(Ctx &c, Kernel kernel, int smem, bool (&set)[64])
{
    static std::mutex mu;
    const int dv = c.device >= 0 && c.device < 64 ? c.device : 0;
    std::lock_guard<std::mutex> lk(mu);
    if (!set[dv]) {
        GALPHA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        set[dv] = true;
    }
    return GPUDT_OK;
}

}  // namespace galpha
