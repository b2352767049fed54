// batch.cu — many independent joins in one persistent, work-stealing launch.
//
// The device-resident form of the reference's block-pair work queue
// (src/queue.cu:142-281, moodycamel ConcurrentQueue + one GPU consumer thread):
// every join of a batch is split into work units (a batch of probes for the
// prefix-index technique, one probe for the exhaustive one and for small
// signature joins; large ones are launches of their own, window.cu);
// the units of all joins form one flat range, and the warps of a single launch
// steal units from it with one atomic each.  A unit finds its join by bisection
// over the units' prefix offsets and runs that join's filter + verify with the
// join's own descriptor (collections, bound tables, index, signatures, output
// buffer), so joins of different sizes, similarity functions, thresholds and
// signature widths share one launch and balance across all 152 SMs.
#include "join_impl.cuh"

namespace hs {

namespace {

// Unit u of a join: a prefix-index join's longest probes go as slot segments
// first (JoinParams::heavy_from), then its probe batches; the window
// techniques' units are single probes.  Items are carried across a unit's slot
// rounds.
template <int W>
__device__ __forceinline__ void run_unit(const BatchDesc& d, uint32_t u, uint32_t* sbuf, int lane) {
    const JoinParams& P = d.P;
    const uint32_t nprobe = P.p_hi - P.p_lo;
    if (d.tech == TECH_FGSS) {
        const uint32_t hf = max(P.heavy_from, P.p_lo), nheavy = P.p_hi > hf ? P.p_hi - hf : 0u;
        uint32_t i0, k, jb = 0, je = 0xFFFFFFFFu;
        if (u < nheavy * P.segs) {
            i0 = u / P.segs;
            k = 1;
            jb = (u - i0 * P.segs) * P.seg_slots;
            je = jb + P.seg_slots;
        } else {
            i0 = nheavy + (u - nheavy * P.segs) * d.unit_probes;
            k = min(d.unit_probes, nprobe - i0);
        }
        ItemCarry ic;
        fgss_carry<1, W, false, false>(P, i0, k, lane, ic, jb, je);
        flush_items<1, W, false, false>(P, ic, lane);
    } else {
        enum_probe<1, W, false>(P, P.p_hi - 1 - u, sbuf, lane);
    }
}

__global__ void __launch_bounds__(JOIN_THREADS, HS_JOIN_MIN_BLOCKS) k_batch_join(const BatchDesc* __restrict__ D,
                                                            const uint32_t* __restrict__ unit_off, uint32_t n_joins,
                                                            unsigned int* work) {
    extern __shared__ uint32_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* sbuf = smem + warp * MAXP;
    const uint32_t total = unit_off[n_joins];
    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = atomicAdd(work, 1u);
        u = __shfl_sync(FULL, u, 0);
        if (u >= total) break;
        uint32_t lo = 0, hi = n_joins;  // the join: largest j with unit_off[j] <= u
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (unit_off[mid] <= u) lo = mid;
            else hi = mid;
        }
        const BatchDesc& d = D[lo];
        u -= unit_off[lo];
        switch (d.words) {
        case 1: run_unit<1>(d, u, sbuf, lane); break;
        case 2: run_unit<2>(d, u, sbuf, lane); break;
        case 4: run_unit<4>(d, u, sbuf, lane); break;
        case 8: run_unit<8>(d, u, sbuf, lane); break;
        default: run_unit<0>(d, u, sbuf, lane); break;
        }
    }
}

}  // namespace

cudaError_t launch_batch_join(const BatchDesc* d_desc, const uint32_t* d_unit_off, uint32_t n_joins,
                              unsigned int* d_work, int sm_count, cudaStream_t s) {
    if (n_joins == 0) return cudaSuccess;
    note_launches();
    const size_t smem = JOIN_WARPS * MAXP * sizeof(uint32_t);
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_join, JOIN_THREADS, smem);
    if (e != cudaSuccess) return e;
    k_batch_join<<<sm_count * (per_sm ? per_sm : 1), JOIN_THREADS, smem, s>>>(d_desc, d_unit_off, n_joins, d_work);
    return cudaGetLastError();
}

}  // namespace hs
