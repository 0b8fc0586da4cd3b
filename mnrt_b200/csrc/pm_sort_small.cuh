// pm_sort_small.cuh -- a whole stable LSD radix sort of up to 65,536
// (key, value) pairs in one launch.
//
// A pass of the multi-kernel sort (pm_sort.cu) is three launches, and below
// some 10^5 keys each costs its launch and drain, not its work: the order of
// 16,384 queries took 13 launches and 64 us, here 22 us with the records laid
// out; 65,536 photons' bounds, codes, sort and move take 63 us in place of 17
// launches and two clears.  Ordering a block's pairs by digit before they leave
// for the other blocks took that build kernel from 74 to 63 us.
// Here one thread-block cluster of up to 16 blocks holds every pair in shared
// memory for the whole sort.  Per 8-bit digit: the blocks rank their pairs
// (warp ballots, counters per warp), publish their 256 digit counts, read the
// other blocks' counts over distributed shared memory after a cluster barrier,
// order their pairs by digit and write them to the blocks that own their
// places; a second barrier ends the pass.  The pairs a thread holds
// sit in registers between the barriers, so one buffer is enough.  The last
// pass hands each pair with its sorted position to the caller's sink instead.
#pragma once

#include <cooperative_groups.h>

#include "pm_internal.h"

namespace pm {

constexpr int kSmallSortThreads = 1024;
constexpr int kSmallSortWarps = kSmallSortThreads / 32;
constexpr uint32_t kSmallSortMaxBlocks = 16;   // above 8 a cluster is a non-portable size: sm_100 allows 16
constexpr uint32_t kSmallSortMax = 65536;      // 4 pairs per thread

struct SmallSortSmem {
    uint16_t cnt[kSmallSortWarps][256];   // per-warp digit counts, then per-warp starts within the block's digit
    uint32_t tot[256];                    // the block's digit counts, read by the whole cluster
    uint32_t base[256];                   // sorted position of the block's first pair of each digit
    uint32_t start[256];                  // the same among the block's own pairs
    uint32_t wsum[2][8];
};

template <class Key, int R>
constexpr int small_sort_smem_bytes() {
    return (int)sizeof(SmallSortSmem) + 2 * kSmallSortThreads * R * (int)(sizeof(Key) + sizeof(uint32_t));
}

// Sorts the cluster's pairs by bits [0, key_bits): this thread's pairs are
// key[r], val[r] at position block * 1024 R + warp * 32 R + 32 r + lane, those
// below n valid.  sink(position, key, value) receives every pair sorted.
template <class Key, int R, class Sink>
__device__ __forceinline__ void small_sort(Key (&key)[R], uint32_t (&val)[R], uint32_t n, int key_bits,
                                           unsigned char* smem, Sink&& sink) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    SmallSortSmem& s = *reinterpret_cast<SmallSortSmem*>(smem);
    constexpr uint32_t per = kSmallSortThreads * R;   // positions of one block (a power of two)
    Key* skey = reinterpret_cast<Key*>(smem + sizeof(SmallSortSmem));   // the block's pairs, written by the cluster
    Key* dkey = skey + per;                                              // its pairs by digit, before they leave
    uint32_t* sval = reinterpret_cast<uint32_t*>(dkey + per);
    uint32_t* dval = sval + per;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    const uint32_t block = cluster.block_rank(), blocks = cluster.num_blocks();
    const uint32_t first = warp * 32u * R + lane;
    const uint32_t mine = block * per < n ? min(per, n - block * per) : 0u;   // valid pairs of the block
    for (int shift = 0; shift < key_bits; shift += 8) {
        const bool last = shift + 8 >= key_bits;
        reinterpret_cast<uint4*>(&s.cnt[0][0])[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        uint32_t rank[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool valid = first + 32u * r < mine;
            const uint32_t digit = (uint32_t)(key[r] >> shift) & 0xffu;
            uint32_t peers = __ballot_sync(0xffffffffu, valid);   // valid lanes with the same digit: 8 ballots
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const uint32_t ones = __ballot_sync(0xffffffffu, (digit >> b) & 1u);
                peers &= ((digit >> b) & 1u) ? ones : ~ones;
            }
            rank[r] = valid ? s.cnt[warp][digit] + __popc(peers & lt) : 0u;
            __syncwarp();
            if (valid && (peers & lt) == 0u) s.cnt[warp][digit] += (uint16_t)__popc(peers);
            __syncwarp();
        }
        __syncthreads();
        if (threadIdx.x < 256) {   // thread d: per-warp starts within digit d, the block's count
            uint32_t run = 0;
#pragma unroll 8
            for (int w = 0; w < kSmallSortWarps; ++w) {
                const uint32_t c = s.cnt[w][threadIdx.x];
                s.cnt[w][threadIdx.x] = (uint16_t)run;
                run += c;
            }
            s.tot[threadIdx.x] = run;
        }
        cluster.sync();   // every block's counts are published, and its pairs are in registers
        uint32_t all = 0, before = 0, x = 0, own = 0, y = 0;
        if (threadIdx.x < 256) {
            for (uint32_t b = 0; b < blocks; ++b) {
                const uint32_t c = cluster.map_shared_rank(&s.tot[0], b)[threadIdx.x];
                all += c;
                before += b < block ? c : 0u;
            }
            own = s.tot[threadIdx.x];
            x = all;   // inclusive scans of the digit totals, the cluster's and the block's
            y = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, x, o), v = __shfl_up_sync(0xffffffffu, y, o);
                if (lane >= (uint32_t)o) { x += u; y += v; }
            }
            if (lane == 31) { s.wsum[0][warp] = x; s.wsum[1][warp] = y; }
        }
        __syncthreads();
        if (threadIdx.x < 256) {
            for (uint32_t w = 0; w < warp; ++w) { x += s.wsum[0][w]; y += s.wsum[1][w]; }
            s.base[threadIdx.x] = x - all + before;
            s.start[threadIdx.x] = y - own;
        }
        __syncthreads();
        // by digit within the block first: runs of equal digits then leave as
        // neighbours, several pairs per transaction between the SMs
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (first + 32u * r >= mine) continue;
            const uint32_t digit = (uint32_t)(key[r] >> shift) & 0xffu;
            const uint32_t local = s.start[digit] + s.cnt[warp][digit] + rank[r];
            dkey[local] = key[r];
            dval[local] = val[r];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t i = threadIdx.x + kSmallSortThreads * r;
            if (i >= mine) continue;
            const Key k = dkey[i];
            const uint32_t v = dval[i], digit = (uint32_t)(k >> shift) & 0xffu;
            const uint32_t dst = s.base[digit] + (i - s.start[digit]);
            if (last) {
                sink(dst, k, v);
            } else {
                cluster.map_shared_rank(skey, dst / per)[dst % per] = k;
                cluster.map_shared_rank(sval, dst / per)[dst % per] = v;
            }
        }
        cluster.sync();   // all pairs delivered (and, after the last pass, no block leaves while its counts are read)
        if (last) break;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (first + 32u * r >= mine) continue;
            key[r] = skey[first + 32u * r];
            val[r] = sval[first + 32u * r];
        }
    }
}

// Blocks of the cluster for n pairs at R per thread: a power of two.
inline uint32_t small_sort_blocks(uint32_t n, int R) {
    const uint32_t per = (uint32_t)(kSmallSortThreads * R);
    uint32_t b = 1;
    while (b * per < n) b <<= 1;
    return b;
}

// Launches `kernel` (which calls small_sort<Key, R>) as one cluster.  False, with
// nothing enqueued and no error left, where that cluster does not fit (up to 16
// blocks of 1,024 threads at once is more than a context limited to part of the
// SMs may have) or the launch is refused: the caller then takes the sort of
// several kernels.  Whether a size fits is asked once and kept in fits, the
// handle's for this kernel (asked on every call: 65,536 photons and 16,384 queries
// 240.5 us in place of 240.0, 4,095 queries 77.7 in place of 77.0).
template <class Key, int R, class... Params, class... Args>
inline bool launch_small_sort(void (*kernel)(Params...), uint32_t n, SmallSortFits& fits, cudaStream_t st, Args... args) {
    constexpr int smem = small_sort_smem_bytes<Key, R>();
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = small_sort_blocks(n, R);
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(at[0].val.clusterDim.x);
    cfg.blockDim = dim3(kSmallSortThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const uint32_t size = (uint32_t)R * 32u + at[0].val.clusterDim.x;   // R at most 4, at most 16 blocks
    bool ok = fits.holds(size);
    if (!ok && !fits.asked(size)) {
        int clusters = 0;
        ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
             cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
             cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0;
        fits.keep(size, ok);
    }
    ok = ok && cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok;
}

}  // namespace pm
