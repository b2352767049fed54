// sort.cu — result pairs put in order in one launch.
//
// A join that returns its pairs sorted mostly has a few hundred to a few ten
// thousand of them, and its time was launches: two stable radix sorts of 32-bit
// keys, 18 to 28 kernels one after the other (70-85 us on GB300 for 8,000 to
// 31,000 pairs, whatever their number).  Here one cluster of eight blocks
// holds every pair as one 64-bit key, (first << second_bits) | second, in its
// shared memory, sorts by digits of at most eight bits and scatters each
// pass through distributed shared memory, so nothing between the passes
// touches memory or waits for a launch.  The bound is the serial chain of a
// pass (the ranking rounds, two cluster barriers): 8 slices x 8,192 keys
// twice (128 KB of a block's 227 KB) is the most that fits beside the
// per-warp digit counts, PAIR_SORT_MAX keys; larger results keep the radix
// sort over memory (sort_pair_list).
#include <cooperative_groups.h>

#include "kernels.h"

namespace cg = cooperative_groups;

namespace hs {

namespace {

constexpr int PS_THREADS = 1024;
constexpr int PS_WARPS = PS_THREADS / 32;
constexpr int PS_CLUSTER = 8;          // the largest portable cluster
constexpr uint32_t PS_SLICE = 8192;    // keys a block holds
constexpr int PS_ROUNDS = PS_SLICE / PS_THREADS;
constexpr int PS_BINS = 256;
static_assert(PAIR_SORT_MAX == (uint64_t)PS_CLUSTER * PS_SLICE, "the cluster holds PAIR_SORT_MAX keys");

struct PairSortSmem {
    uint64_t key[2][PS_SLICE];
    uint32_t whist[PS_WARPS][PS_BINS];  // per-warp digit counts, then their exclusive sums over the warps
    uint32_t total[PS_BINS];            // the block's digit counts (read by the whole cluster)
    uint32_t base[PS_BINS];             // where the block's keys of each digit go
    uint32_t wsum[PS_BINS / 32];
};

// One cluster per job.  Slice c of the keys (2^mshift of them, a power of two)
// lies in block c; a warp owns consecutive keys of its slice and ranks them 32
// at a time, so the sort is stable.
__global__ void __cluster_dims__(PS_CLUSTER, 1, 1) __launch_bounds__(PS_THREADS, 1)
    k_sort_pairs(PairSortJob one, const PairSortJob* __restrict__ jobs) {
    extern __shared__ __align__(16) uint8_t pair_sort_smem[];
    PairSortSmem& sm = *reinterpret_cast<PairSortSmem*>(pair_sort_smem);
    cg::cluster_group cluster = cg::this_cluster();
    const PairSortJob J = jobs ? jobs[blockIdx.x / PS_CLUSTER] : one;
    const unsigned long long count = *J.count;
    if (count <= 1 || count > J.cap || count > PAIR_SORT_MAX) return;  // the whole cluster
    const uint32_t n = (uint32_t)count;
    const uint32_t c = cluster.block_rank();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t mshift = 5;
    while (((uint64_t)PS_CLUSTER << mshift) < n) ++mshift;
    const uint32_t m = 1u << mshift;
    const uint32_t lo = c << mshift;
    const uint32_t mine = n > lo ? min(m, n - lo) : 0u;        // keys of this slice
    const uint32_t rounds = max(1u, m / PS_THREADS);           // of 32 keys per warp
    const uint32_t w0 = (uint32_t)warp * 32u * rounds;         // the warp's first key
    uint2* pairs = J.pairs + lo;
    for (uint32_t i = threadIdx.x; i < mine; i += PS_THREADS) {
        const uint2 p = pairs[i];
        sm.key[0][i] = ((uint64_t)p.x << J.second_bits) | p.y;
    }
    const int bits = J.first_bits + J.second_bits;
    const int passes = (bits + 7) / 8, width = (bits + passes - 1) / passes;
    const uint32_t mask = (1u << width) - 1u;
    int cur = 0;
    for (int p = 0; p < passes; ++p, cur ^= 1) {
        const int shift = p * width;
        uint4* z = reinterpret_cast<uint4*>(&sm.whist[0][0]);
        for (uint32_t q = threadIdx.x; q < PS_WARPS * PS_BINS / 4; q += PS_THREADS) z[q] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        uint64_t k[PS_ROUNDS];
        uint32_t rank[PS_ROUNDS];
#pragma unroll
        for (int r = 0; r < PS_ROUNDS; ++r) {
            if (r < (int)rounds) {
                const uint32_t i = w0 + 32u * r + lane;
                const bool valid = i < mine;
                k[r] = valid ? sm.key[cur][i] : 0ull;
                const uint32_t d = (uint32_t)(k[r] >> shift) & mask;
                // the lanes with this digit, by a vote per bit (__match_any_sync took
                // several times as long: 128 of them per block and pass)
                unsigned peers = __ballot_sync(FULL, valid);
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    const unsigned set = __ballot_sync(FULL, (d >> b) & 1u);
                    peers &= (d >> b) & 1u ? set : ~set;
                }
                const uint32_t before = valid ? sm.whist[warp][d] : 0u;
                __syncwarp();
                if (valid && lane == __ffs(peers) - 1) sm.whist[warp][d] = before + __popc(peers);
                __syncwarp();
                rank[r] = before + __popc(peers & lanemask_lt(lane));
            }
        }
        __syncthreads();
        if (threadIdx.x < PS_BINS) {
            uint32_t acc = 0;
#pragma unroll 8
            for (int w = 0; w < PS_WARPS; ++w) {
                const uint32_t x = sm.whist[w][threadIdx.x];
                sm.whist[w][threadIdx.x] = acc;
                acc += x;
            }
            sm.total[threadIdx.x] = acc;
        }
        cluster.sync();
        uint32_t all = 0, before = 0, incl = 0;
        if (threadIdx.x < PS_BINS) {
#pragma unroll
            for (uint32_t b = 0; b < PS_CLUSTER; ++b) {
                const uint32_t x = cluster.map_shared_rank(sm.total, b)[threadIdx.x];
                all += x;
                before += b < c ? x : 0u;
            }
            incl = warp_incl_scan(all, lane);
            if (lane == 31) sm.wsum[warp] = incl;
        }
        __syncthreads();
        if (threadIdx.x < PS_BINS) {
            uint32_t at = incl - all + before;
#pragma unroll
            for (int w = 0; w < PS_BINS / 32; ++w) at += w < warp ? sm.wsum[w] : 0u;
            sm.base[threadIdx.x] = at;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < PS_ROUNDS; ++r) {
            if (r < (int)rounds && w0 + 32u * r + lane < mine) {
                const uint32_t d = (uint32_t)(k[r] >> shift) & mask;
                const uint32_t at = sm.base[d] + sm.whist[warp][d] + rank[r];
                cluster.map_shared_rank(sm.key[cur ^ 1], at >> mshift)[at & (m - 1u)] = k[r];
            }
        }
        cluster.sync();
    }
    const uint32_t low = J.second_bits >= 32 ? 0xFFFFFFFFu : (1u << J.second_bits) - 1u;
    for (uint32_t i = threadIdx.x; i < mine; i += PS_THREADS) {
        const uint64_t key = sm.key[cur][i];
        pairs[i] = make_uint2((uint32_t)(key >> J.second_bits), (uint32_t)key & low);
    }
}

}  // namespace

cudaError_t prepare_sort_kernels() {
    return cudaFuncSetAttribute(k_sort_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PairSortSmem));
}

cudaError_t sort_pairs_cluster(const PairSortJob& job, cudaStream_t s) {
    note_launches();
    k_sort_pairs<<<PS_CLUSTER, PS_THREADS, sizeof(PairSortSmem), s>>>(job, nullptr);
    return cudaGetLastError();
}

cudaError_t sort_pairs_clusters(const PairSortJob* d_jobs, uint32_t n_jobs, cudaStream_t s) {
    if (n_jobs == 0) return cudaSuccess;
    note_launches();
    k_sort_pairs<<<PS_CLUSTER * n_jobs, PS_THREADS, sizeof(PairSortSmem), s>>>(PairSortJob{}, d_jobs);
    return cudaGetLastError();
}

}  // namespace hs
