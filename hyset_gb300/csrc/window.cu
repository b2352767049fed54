// window.cu — the signature (bitmap) technique: every length-compatible pair's
// XOR signatures compared, the survivors verified (replaces bitmap::filter,
// include/hyset/device_algorithms.hpp:76-118, and verify_pairs).
//
// What bounds it: the pairs of all length windows (6.5e9 for 200,000 short
// sets at Jaccard 0.7) times the instructions one pair costs; memory is read
// once per tile and served from L2.  A warp per probe that walked its window
// (enum_probe, join_impl.cuh) spent about 75 issue slots on a pair: its
// candidate's record, its bound, its signature's loads and a vote each time.
// Here a block holds a tile of up to 64 consecutive probes in shared memory
// and each lane NC candidates' signatures in registers, so a pair costs its
// XORs, a population count and a shift:
//   - sets are ordered by size, so the largest admissible distance
//     |r| + |s| - 2 minoverlap is one value per (lane, candidate) until the
//     probe's size changes; a candidate outside the size window gets none;
//   - POPC runs at a quarter of the logic rate, so the words are first OR-ed
//     into G groups: popc(x0 | x1 | ...) <= the distance, so a pair rejected
//     by the groups' counts is rejected by the distance.  G follows from the
//     admissible distance: a group can count to 32 at most, and pairs of
//     unrelated sets fill three quarters of the bits of two dense words;
//   - eight probes' outcomes are collected as sign bits in one mask, and only
//     a mask that is not zero leaves the loop: its pairs are checked exactly
//     (window, distance over all words) and queued, and 32 queued pairs are
//     verified at a time, a lane or the warp each.
// 200,000 short sets (lognormal, mean 29), Jaccard 0.7, 64 bits on GB300: a
// call 13.76 ms before, 2.40 ms with this kernel alone, 1.93 with its longest
// probes in launches of wider signatures (widen_window, join_host.cu).  Alone:
// one block fewer per SM for W <= 2 2.52, heavy probes (see WinCut) 4 / 8 to a
// unit 2.70 / 2.52, segments of 4,096 2.58, one group up to a distance of 14 or
// 18 instead of 16 within 1 %.
#include "join_impl.cuh"

namespace hs {

namespace {

constexpr int WIN_THREADS = 256;
constexpr int WIN_WARPS = WIN_THREADS / 32;
constexpr uint32_t WIN_TILE = 64;   // probes a block holds
constexpr uint32_t WIN_GROUP = 8;   // probes between two looks at the mask
constexpr uint32_t WIN_QUEUE = 64;  // pairs waiting for verification, per warp (31 + 32 at most)

template <int W>
__host__ __device__ constexpr int win_cands() {  // candidates per lane
    return W <= 2 ? 4 : 2;
}

template <int W>
struct WinSmem {
    uint32_t sig[WIN_TILE][2 * W];  // the probes' signatures
    uint32_t len[WIN_TILE];
    uint2 queue[WIN_WARPS][WIN_QUEUE];
    uint32_t unit;
};

// One more than the largest admissible signature distance of a pair of sizes
// lp (probe) and lc (candidate); 0 when the candidate is outside the probe's
// size window.
__device__ __forceinline__ int distance_limit(const JoinParams& P, uint32_t lp, uint32_t lc) {
    if (lc == 0 || lc < P.B.minsize[lp] || lc > (P.self ? lp : P.B.max_partner[lp])) return 0;
    return (int)(lp + lc + 1u) - 2 * (int)minoverlap(P.B, max(lp, lc), min(lp, lc));
}

// Eight probes against the lane's candidates: bit 8 NC - 1 - (k NC + j) of the
// result is set where the G groups' counts leave probe k and candidate j in.
template <int W, int G>
__device__ __forceinline__ uint32_t compare_group(const uint32_t (*sig)[2 * W], const uint32_t (&cw)[win_cands<W>()][2 * W],
                                                  const int (&lim)[win_cands<W>()]) {
    constexpr int NW = 2 * W, NC = win_cands<W>();
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < (int)WIN_GROUP; ++k) {
        uint32_t pw[NW];
#pragma unroll
        for (int w = 0; w < NW; w += 2) {
            const uint2 v = *reinterpret_cast<const uint2*>(&sig[k][w]);
            pw[w] = v.x;
            pw[w + 1] = v.y;
        }
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            int pop = 0;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                uint32_t x = cw[j][g] ^ pw[g];
#pragma unroll
                for (int w = g + G; w < NW; w += G) x |= cw[j][w] ^ pw[w];
                pop += __popc(x);
            }
            m = __funnelshift_l((uint32_t)(pop - lim[j]), m, 1);
        }
    }
    return m;
}

// Verifies the warp's first n queued pairs (n <= 32), a lane or the warp each.
template <int VMODE>
__device__ __forceinline__ void verify_queued(const JoinParams& P, const uint2* queue, uint32_t n, int lane) {
    const bool has = (uint32_t)lane < n;
    uint2 it = make_uint2(0, 0), pm = make_uint2(0, 0), cm = make_uint2(0, 0);
    uint32_t mo = 0;
    if (has) {
        it = queue[lane];
        pm = P.S.meta[it.x];
        cm = P.R.meta[it.y];
        mo = minoverlap(P.B, max(pm.y, cm.y), min(pm.y, cm.y));
    }
    if constexpr (VMODE == 1) {
        const bool ok = has && verify_serial(P.S.tokens + pm.x, pm.y, P.R.tokens + cm.x, cm.y, mo, NOWN);
        emit(P.out, ok, it.x, it.y, lane);
    } else {
        bool mine = false;
        for (int src = 0; src < (int)n; ++src) {
            const uint32_t ps = __shfl_sync(FULL, pm.x, src), pl = __shfl_sync(FULL, pm.y, src);
            const uint32_t cs = __shfl_sync(FULL, cm.x, src), cl = __shfl_sync(FULL, cm.y, src);
            const bool ok = verify_warp(P.S.tokens + ps, pl, P.R.tokens + cs, cl, __shfl_sync(FULL, mo, src), NOWN, lane);
            if (lane == src) mine = ok;
        }
        emit(P.out, mine, it.x, it.y, lane);
    }
}

// How probes [p_lo, p_hi) and their windows are cut into units.
struct WinCut {
    uint32_t tile, seg, segs;  // probes and candidates per unit, units per tile of probes
};

// Units (tile of probes) x (segment of its window's candidates) are taken one
// per steal, the longest sets first; a unit past the end of its tile's window
// is empty.  Probes from heavy_from on are cut finer: their signatures are
// full, so most pairs are verified, a merge of long sets each, and a unit of
// 64 x 8,192 of them outlasted the rest of the launch (SMs active 47 % of
// it at 64 bits and 200,000 short sets).
template <int VMODE, int W>
__global__ void __launch_bounds__(WIN_THREADS, W <= 2 ? 5 : 4) k_window(JoinParams P, WinCut heavy, WinCut rest) {
    constexpr int NW = 2 * W, NC = win_cands<W>();
    static_assert(WIN_GROUP * NC <= 32, "a group's outcomes fill one mask");
    __shared__ __align__(16) WinSmem<W> sm;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint2* queue = sm.queue[warp];
    uint32_t qn = 0;  // queued pairs (warp-uniform)
    const uint32_t split = max(P.p_lo, min(P.p_hi, P.heavy_from));  // probes [split, p_hi) are the heavy ones
    const uint32_t units_heavy = (P.p_hi - split + heavy.tile - 1) / heavy.tile * heavy.segs;
    const uint32_t units = units_heavy + (split - P.p_lo + rest.tile - 1) / rest.tile * rest.segs;
    const uint32_t* __restrict__ sig_R = reinterpret_cast<const uint32_t*>(P.bits_R);
    const uint32_t* __restrict__ sig_S = reinterpret_cast<const uint32_t*>(P.bits_S);
    for (;;) {
        __syncthreads();  // the previous unit's tile is no longer read
        if (threadIdx.x == 0) sm.unit = atomicAdd(P.work, 1u);
        __syncthreads();
        uint32_t u = sm.unit;
        if (u >= units) break;
        const bool hv = u < units_heavy;
        if (!hv) u -= units_heavy;
        const WinCut cut = hv ? heavy : rest;
        const uint32_t tile = u / cut.segs, s = u - tile * cut.segs;
        const uint32_t p_end = (hv ? P.p_hi : split) - tile * cut.tile;
        const uint32_t np = min(cut.tile, p_end - (hv ? split : P.p_lo)), p0 = p_end - np;
        const uint32_t lmin = P.S.meta[p0].y, lmax = P.S.meta[p_end - 1].y;
        // the union of the tile's windows (minsize and max_partner grow with the size)
        const uint32_t lo = max(P.first_ge[min(P.B.minsize[lmin], P.R_L + 1)], P.r_lo);
        const uint32_t hi = min(P.self ? p_end - 1 : P.first_ge[min(P.B.max_partner[lmax] + 1, P.R_L + 1)], P.r_hi);
        const uint64_t a64 = (uint64_t)(lo & ~31u) + (uint64_t)s * cut.seg;
        if (a64 >= hi) continue;
        const uint32_t a = (uint32_t)a64, b = (uint32_t)min((uint64_t)hi, a64 + cut.seg);
        for (uint32_t i = threadIdx.x; i < WIN_TILE * NW; i += WIN_THREADS)
            sm.sig[0][i] = i < np * NW ? sig_S[(uint64_t)p0 * NW + i] : 0u;
        for (uint32_t i = threadIdx.x; i < WIN_TILE; i += WIN_THREADS) sm.len[i] = P.S.meta[p0 + min(i, np - 1)].y;
        __syncthreads();
        for (uint32_t c0 = a + (uint32_t)warp * 32u * NC; c0 < b; c0 += WIN_WARPS * 32u * NC) {
            uint32_t cw[NC][NW], lc[NC];
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const uint32_t c = c0 + 32u * j + lane;
                const bool in = c < b;
                lc[j] = in ? P.R.meta[c].y : 0u;
#pragma unroll
                for (int w = 0; w < NW; w += 2) {
                    const uint2 v = in ? __ldg(reinterpret_cast<const uint2*>(sig_R + (uint64_t)c * NW + w))
                                       : make_uint2(0u, 0u);
                    cw[j][w] = v.x;
                    cw[j][w + 1] = v.y;
                }
            }
            int lim[NC], most = 0;  // per candidate, and the warp's largest
            uint32_t cur = 0xFFFFFFFFu;  // the probe size they are for
            auto limits = [&](uint32_t lp) {
                if (lp == cur) return;
                cur = lp;
                most = 0;
#pragma unroll
                for (int j = 0; j < NC; ++j) {
                    lim[j] = distance_limit(P, lp, lc[j]);
                    most = max(most, lim[j]);
                }
                most = __reduce_max_sync(FULL, most);
            };
            for (uint32_t k0 = 0; k0 < np; k0 += WIN_GROUP) {
                uint32_t m = 0;
                if (sm.len[k0] == sm.len[k0 + WIN_GROUP - 1]) {  // sizes ascend: one size
                    limits(sm.len[k0]);
                    if (most == 0) continue;
                    const uint32_t(*sig)[NW] = &sm.sig[k0];
                    // the fewest counts that still reject unrelated dense sets (group limits 24, 48, 96, 192, less
                    // two to three standard deviations)
                    if (most <= 17) m = compare_group<W, 1>(sig, cw, lim);
                    else if (NW > 2 && most <= 41) m = compare_group<W, NW >= 2 ? 2 : 1>(sig, cw, lim);
                    else if (NW > 4 && most <= 85) m = compare_group<W, NW >= 4 ? 4 : 1>(sig, cw, lim);
                    else if (NW > 8 && most <= 173) m = compare_group<W, NW >= 8 ? 8 : 1>(sig, cw, lim);
                    else m = compare_group<W, NW>(sig, cw, lim);
                } else {
#pragma unroll 1
                    for (uint32_t k = 0; k < WIN_GROUP; ++k) {
                        limits(sm.len[k0 + k]);
#pragma unroll
                        for (int j = 0; j < NC; ++j) {
                            int pop = 0;
#pragma unroll
                            for (int w = 0; w < NW; ++w) pop += __popc(cw[j][w] ^ sm.sig[k0 + k][w]);
                            m = __funnelshift_l((uint32_t)(pop - lim[j]), m, 1);
                        }
                    }
                }
                if (np - k0 < WIN_GROUP) m &= ~((1u << ((WIN_GROUP - (np - k0)) * NC)) - 1u);  // no probe there
                while (__any_sync(FULL, m != 0)) {
                    bool keep = m != 0;
                    uint32_t p = 0, c = 0;
                    if (keep) {
                        const int bit = 31 - __clz(m);
                        m &= ~(1u << bit);
                        const uint32_t i = WIN_GROUP * NC - 1 - bit, k = k0 + i / NC;
                        p = p0 + k;
                        c = c0 + 32u * (i % NC) + lane;
                        keep = k < np && c < b;
                        if (keep) {
                            const uint32_t lp = sm.len[k];
                            const Window win = candidate_window(P, p, lp);
                            keep = c >= win.lo && c < win.hi;
                            if (keep) {
                                uint32_t pop = 0;
#pragma unroll
                                for (int w = 0; w < NW; ++w) pop += __popc(sm.sig[k][w] ^ __ldg(sig_R + (uint64_t)c * NW + w));
                                const uint32_t l = P.R.meta[c].y;
                                keep = lp + l - pop >= 2u * minoverlap(P.B, max(lp, l), min(lp, l));
                            }
                        }
                    }
                    const unsigned q = __ballot_sync(FULL, keep);
                    if (keep) queue[qn + __popc(q & lanemask_lt(lane))] = make_uint2(p, c);
                    qn += __popc(q);
                    __syncwarp();
                    if (qn >= 32) {
                        verify_queued<VMODE>(P, queue, 32, lane);
                        qn -= 32;
                        const uint2 rest = (uint32_t)lane < qn ? queue[32 + lane] : make_uint2(0, 0);
                        __syncwarp();
                        if ((uint32_t)lane < qn) queue[lane] = rest;
                        __syncwarp();
                    }
                }
            }
        }
    }
    if (qn) verify_queued<VMODE>(P, queue, qn, lane);
}

template <int VMODE, int W>
cudaError_t launch_window_w(const JoinParams& P, int sm_count, cudaStream_t s) {
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_window<VMODE, W>, WIN_THREADS, 0);
    if (e != cudaSuccess) return e;
    const uint32_t blocks = (uint32_t)(sm_count * std::max(per_sm, 1));
    const uint64_t ncand = P.r_hi > P.r_lo ? P.r_hi - P.r_lo : 1;
    const uint32_t split = std::max(P.p_lo, std::min(P.p_hi, P.heavy_from));
    auto segments = [](uint64_t cands, uint32_t seg) { return (cands + 31 + seg - 1) / seg; };  // a window starts up to 31 ids early
    auto units = [&](uint64_t probes, uint64_t cands, uint32_t tile, uint32_t seg) {
        return (probes + tile - 1) / tile * segments(cands, seg);
    };
    // units small enough that the blocks have several each: down to 16 probes x 1,024
    // candidates, the heavy probes' down to one x 1,024 (below)
    WinCut rest{WIN_TILE, 8192, 0}, heavy{16, 1024, 0};
    const uint64_t np = split - P.p_lo, nh = P.p_hi - split;
    const uint64_t hcand = P.r_hi > std::max(P.r_lo, P.heavy_lo) ? P.r_hi - std::max(P.r_lo, P.heavy_lo) : 1;
    while (units(np, ncand, rest.tile, rest.seg) < 8ull * blocks && rest.seg > 1024) rest.seg /= 2;
    while (units(np, ncand, rest.tile, rest.seg) < 8ull * blocks && rest.tile > 16) rest.tile /= 2;
    // the heavy ones' pairs are mostly verified: down to four probes for a tail of
    // a thirtieth of the launch, to one when there are fewer units than blocks take
    // (8,000 long sets at 128 bits: a thousand heavy probes in 63 units of 16 took
    // 0.6 ms; 30,000 at 64 bits, cosine 0.9: 1.08 ms at 16 to a unit, 0.71 at four)
    while (nh && units(nh, hcand, heavy.tile, heavy.seg) < 32ull * blocks && heavy.tile > 4) heavy.tile /= 2;
    while (nh && units(nh, hcand, heavy.tile, heavy.seg) < 8ull * blocks && heavy.tile > 1) heavy.tile /= 2;
    while (units(np, ncand, rest.tile, rest.seg) > 0x7FFF0000ull) rest.seg *= 2;  // the steal counter has 32 bits
    while (units(nh, hcand, heavy.tile, heavy.seg) > 0x7FFF0000ull) heavy.seg *= 2;
    rest.segs = (uint32_t)segments(ncand, rest.seg);
    heavy.segs = (uint32_t)segments(hcand, heavy.seg);
    const uint64_t all = units(np, ncand, rest.tile, rest.seg) + units(nh, hcand, heavy.tile, heavy.seg);
    note_launches();
    k_window<VMODE, W><<<(unsigned)std::min<uint64_t>(blocks, all), WIN_THREADS, 0, s>>>(P, heavy, rest);
    return cudaGetLastError();
}

template <int VMODE>
cudaError_t launch_window_v(const JoinParams& P, int sm_count, cudaStream_t s) {
    switch (P.words) {
    case 1: return launch_window_w<VMODE, 1>(P, sm_count, s);
    case 2: return launch_window_w<VMODE, 2>(P, sm_count, s);
    case 4: return launch_window_w<VMODE, 4>(P, sm_count, s);
    case 8: return launch_window_w<VMODE, 8>(P, sm_count, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t launch_window(const JoinParams& P, int vmode, int sm_count, cudaStream_t s) {
    return vmode == 2 ? launch_window_v<2>(P, sm_count, s) : launch_window_v<1>(P, sm_count, s);
}

}  // namespace hs
