// join_host.cu — one join: technique and configuration, index and
// signatures, the persistent filter + verify launch (re-run once with an
// exact buffer when the pairs overflowed), the optional device sort of the
// pairs, and the self-join / R-S join entry points.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>

#include "host.h"

namespace hs {

// Orders n result pairs by (probe id, indexed id) on the device, in place.
hyset_status sort_device_pairs(hyset_ctx* ctx, uint2* pairs, uint64_t n, uint32_t n_probe, uint32_t n_indexed) {
    if (n <= 1) return HYSET_OK;
    cudaStream_t s = ctx->stream;
    Scratch& sc = ctx->own;
    const size_t b = (size_t)n * 4;
    CK(sc.tok.ensure(b, s));
    CK(sc.set.ensure(b, s));
    CK(sc.altk.ensure(b, s));
    CK(sc.altv.ensure(b, s));
    CK(sc.scan.ensure(radix_scratch_words(n) * 4, s));
    CK(sort_pair_list(pairs, n, (int)bits_for(n_probe), (int)bits_for(n_indexed), sc.tok.as<uint32_t>(),
                      sc.set.as<uint32_t>(), sc.altk.as<uint32_t>(), sc.altv.as<uint32_t>(), sc.scan.as<uint32_t>(),
                      s));
    return HYSET_OK;
}

// R-S joins are symmetric in the two collections (the bounds take the larger
// and smaller size of a pair, both sides keep maxprefix tokens), so the
// collections' roles may be exchanged: the indexed side is the smaller one
// (a cheaper index build) and the probe side the larger one (more work units
// for the persistent launch).  Output pairs are written back in the caller's
// (probe, indexed) order.  Probe ranges shard the caller's probe side and keep
// the given orientation.
bool swap_sides(const hyset_coll* R, const hyset_coll* S, const hyset_join_opts* o) {
    if (R == S || o->probe_end) return false;
    if (o->orientation == 2) return true;
    return o->orientation == 0 && S->n < R->n;
}

// Runs one configured join launch into the context's pair buffer, growing the
// buffer and re-running when the first pass overflowed.
hyset_status run_join(hyset_ctx* ctx, JoinParams P, int tech, int vmode, const hyset_join_opts* o,
                      hyset_result* res, bool timed_from_ev0, TokenJoinParams* T,
                      const std::vector<JoinParams>* parts) {
    cudaStream_t s = ctx->stream;
    const int count_only = o->count_only ? 1 : 0;
    uint64_t cap = o->pair_capacity ? o->pair_capacity : std::max<uint64_t>(1u << 20, 4ull * P.S.n);
    if (count_only) cap = 0;
    CK(ctx->s_count.ensure(32, s));  // the count, then the launch's counters: one clear
    CK(ctx->s_stats.ensure(64, s));
    P.stats = o->collect_stats ? ctx->s_stats.as<unsigned long long>() : nullptr;
    for (int attempt = 0; attempt < 2; ++attempt) {
        if (!count_only) CK(ctx->s_pairs.ensure(std::max<uint64_t>(cap, 1) * sizeof(uint2), s));
        P.out.pairs = count_only ? nullptr : ctx->s_pairs.as<uint2>();
        P.out.count = ctx->s_count.as<unsigned long long>();
        P.out.cap = cap;
        P.out.count_only = count_only;
        P.work = ctx->s_count.as<unsigned int>() + 4;
        if (!timed_from_ev0 || attempt > 0) CK(cudaEventRecord(ctx->ev0, s));
        CK(cudaMemsetAsync(ctx->s_count.p, 0, 32, s));
        if (P.stats) CK(cudaMemsetAsync(P.stats, 0, 64, s));
        CK(cudaEventRecord(ctx->ek0, s));
        if (T) {
            T->out = P.out;
            T->work = P.work;
            T->stats = P.stats;
            CK(launch_join_tm(*T, ctx->sm_count, s));
        } else if (parts && !parts->empty()) {  // up to three launches, a counter each
            for (size_t k = 0; k < parts->size(); ++k) {
                JoinParams Q = (*parts)[k];
                Q.out = P.out;
                Q.work = P.work + k;
                CK(launch_join(Q, tech, vmode, ctx->sm_count, s));
            }
        } else {
            CK(launch_join(P, tech, vmode, ctx->sm_count, s));
        }
        CK(cudaEventRecord(ctx->ek1, s));
        CK(cudaEventRecord(ctx->ev1, s));
        ST(enqueue_result(ctx, P, o));
        if (P.stats) CK(cudaMemcpyAsync(res->stats, P.stats, 64, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        const uint64_t count = joined_count(ctx);
        float ms = 0, kms = 0;
        CK(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
        CK(cudaEventElapsedTime(&kms, ctx->ek0, ctx->ek1));
        res->device_ms = ms;
        res->kernel_ms = kms;
        res->count = count;
        if (count_only || count <= cap) break;
        cap = count + count / 8 + 1024;  // overflow: retry once with room for everything
        if (attempt == 1) return fail(ctx, HYSET_E_OVERFLOW, "pair buffer overflow after resize");
    }
    return deliver_pairs(ctx, P, o, res);
}

// A probe of a long prefix is one warp's work: unsplit, the longest probes of
// the 61,003 x 147,001 dice join at 0.75 (1,400 slots in two bands) held the
// launch for twice its other warps' time (kernel 0.79 ms at its best batch of
// one probe, 1.04 at three; 0.47 split).  Above 64 / 96 / 128 slots, a call of
// that join: 0.865 / 0.789 / 0.776 ms; units of 32 / 64 / 128 slots 0.809 /
// 0.776 / 0.801.
// The units are a grid, split probes x segments of the longest prefix, counted
// in 32 bits, and most of it is empty where one set is far longer than the
// others: a set of 4,200,000 tokens beside 131,200 of 260 made 2^32 + 10^7 units
// of 64 slots at Jaccard 0.5, and the probes of the first 2^32 were left out.  So
// the segments grow until the grid is at most four times what the probes' own
// slots fill (32 million units, whatever they are; a million always pass).
void split_heavy(const hyset_coll* S, const Bounds* b, JoinParams& P) {
    constexpr uint32_t HEAVY_SLOTS = 128;  // probes with longer prefixes are split
    constexpr uint32_t SEG_SLOTS = 64;     // prefix slots per unit of a split probe
    constexpr uint64_t MANY_UNITS = 1ull << 20, MOST_UNITS = 1ull << 25;  // 2^32 tokens hold 2^24 split probes at most
    P.heavy_from = 0xFFFFFFFFu;
    P.segs = 0;
    P.seg_slots = SEG_SLOTS;
    const uint32_t L = std::min(S->max_size, b->L);
    for (uint32_t l = 0; l <= L; ++l)
        if (b->probe_prefix[l] > HEAVY_SLOTS) {
            P.heavy_from = S->h_first_ge[l];
            P.segs = (b->probe_prefix[L] + SEG_SLOTS - 1) / SEG_SLOTS;
            const uint64_t heavy = S->n - P.heavy_from;
            if (heavy * P.segs <= MANY_UNITS) return;
            uint64_t filled = heavy;
            for (uint32_t k = l; k <= L; ++k) filled += S->size_hist[k] * (uint64_t)b->probe_prefix[k] / SEG_SLOTS;
            const uint64_t most = std::min(std::max(4 * filled, MANY_UNITS), MOST_UNITS);
            while (heavy * P.segs > most) {
                P.seg_slots *= 2;
                P.segs = (b->probe_prefix[L] + P.seg_slots - 1) / P.seg_slots;
            }
            return;
        }
}

static int width_index(int words) { return words >= 8 ? 3 : words >= 4 ? 2 : words >= 2 ? 1 : 0; }

// The first size whose equally long pairs may differ in three eighths of the
// signature: two sets of many tokens differ in half of its bits, give or take
// sqrt(bits) / 2, so from there on unrelated pairs start to pass (64 bits: at
// 24, two deviations short of 32).  Kept with the bound tables, as filled_from
// is: the searches of each call took 4-7 us of a call on 2,000 long sets
// (128 bits, Jaccard 0.8: 103 -> 96 us).
static uint32_t split_from(const Bounds* b, int words) {
    uint32_t& size = b->split_size[width_index(words)];
    if (size) return size;
    const uint32_t least = 64u * (uint32_t)words * 3 / 8;
    uint32_t l = 1;
    while (l <= b->L && 2 * l - 2 * minoverlap_of(b->sim, l, l, b->tau) < least) ++l;
    return size = l;
}

void split_window(const hyset_coll* R, const hyset_coll* S, const Bounds* b, int words, JoinParams& P) {
    P.heavy_from = 0xFFFFFFFFu;
    const uint32_t l = split_from(b, words);
    if (l > std::min(S->max_size, b->L)) return;
    P.heavy_from = S->h_first_ge[l];
    P.heavy_lo = R->h_first_ge[std::min(b->minsize[l], R->max_size + 1)];
}

// The size from which on unrelated pairs of one size pass signatures of `words`
// words: two sets of l tokens differ in about E = bits / 2 (1 - exp(-4 l / bits))
// bits, and from an admissible distance of E less two deviations on more than a
// few percent pass.
static uint32_t filled_from(const Bounds* b, int words) {
    uint32_t& size = b->filled_size[width_index(words)];
    if (size) return size;
    const double bits = 64.0 * words;
    uint32_t l = b->L + 1;
    for (; l > 1; --l) {
        const double e = 0.5 * bits * (1.0 - std::exp(-4.0 * (l - 1) / bits));
        const uint32_t most = 2 * (l - 1) - 2 * minoverlap_of(b->sim, l - 1, l - 1, b->tau);
        if ((double)most < e - 2.0 * std::sqrt(e * (1.0 - e / bits))) break;
    }
    return size = l;
}

// Pairs that pass a full signature are all verified, 5 ps each and more for
// long sets (200,000 short sets at 64 bits, Jaccard 0.5: 1.2e10 pairs in 61 ms),
// where a signature that still rejects costs a pair 0.3 ps (64 bits) to 1.2
// (512).  So the probes that fill their signatures take 256 bits, and those that
// fill these 512; WIDE_PAIRS pairs cost their verification about what a width's
// generation and launch cost (at half as many, joins of 8,000 long sets lost
// 10 to 20 us; with 128 bits between 64 and 256, 100,000 long sets took 3.3 ms
// instead of 2.8 at cosine 0.75).
void cut_window(const hyset_coll* R, const hyset_coll* S, const Bounds* b, const JoinParams& P,
                std::vector<JoinParams>& parts) {
    constexpr uint64_t WIDE_PAIRS = 16ull << 20;
    parts.assign(1, P);
    for (int words = std::max(4, 2 * P.words); words <= 8; words *= 2) {
        if ((uint64_t)(P.p_hi - P.p_lo) * R->n < WIDE_PAIRS) break;
        const uint32_t filled = filled_from(b, parts.back().words);
        const uint32_t from = filled > S->max_size ? P.p_hi : std::max(P.p_lo, std::min(P.p_hi, S->h_first_ge[filled]));
        if (from >= P.p_hi) break;
        const uint32_t least = std::min(b->minsize[size_at(S, from)], R->max_size + 1);
        if ((uint64_t)(P.p_hi - from) * (R->n - R->h_first_ge[least]) < WIDE_PAIRS) break;
        JoinParams W = P;
        W.bits_R = W.bits_S = nullptr;
        W.words = words;
        W.p_lo = from;
        split_window(R, S, b, words, W);
        parts.back().p_hi = from;
        parts.push_back(W);
    }
}

void drop_widest(std::vector<JoinParams>& parts) {
    const uint32_t hi = parts.back().p_hi;
    parts.pop_back();
    parts.back().p_hi = hi;
}

void order_widths(std::vector<JoinParams>& parts) {
    std::reverse(parts.begin(), parts.end());  // the longest sets first
    parts.erase(std::remove_if(parts.begin(), parts.end(), [](const JoinParams& q) { return q.p_lo >= q.p_hi; }),
                parts.end());
}

hyset_status widen_window(hyset_ctx* ctx, hyset_coll* R, hyset_coll* S, const Bounds* b, const JoinParams& P,
                          cudaStream_t gen, std::vector<JoinParams>& parts) {
    cut_window(R, S, b, P, parts);
    auto room = [&](hyset_coll* c, int words) {
        return c->bitmaps[words].ensure(sig_bytes(c->n, words), ctx->stream) == cudaSuccess;
    };
    for (size_t k = 1; k < parts.size(); ++k) {
        JoinParams& W = parts[k];
        if (!room(R, W.words) || (S != R && !room(S, W.words))) {  // without room for them the narrow ones do
            while (parts.size() > k) drop_widest(parts);
            break;
        }
        const uint64_t *br = nullptr, *bs = nullptr;
        ST(get_bitmaps(ctx, R, W.words, &br, gen));
        if (S == R) bs = br;
        else ST(get_bitmaps(ctx, S, W.words, &bs, gen));
        W.bits_R = br;
        W.bits_S = bs;
    }
    if (parts.size() == 1) parts.clear();
    order_widths(parts);
    return HYSET_OK;
}

PairSortJob pair_sort_job(const JoinParams& P) {
    return PairSortJob{P.out.pairs, P.out.count, P.out.cap, (int)bits_for(P.out.swap ? P.R.n : P.S.n),
                       (int)bits_for(P.out.swap ? P.S.n : P.R.n)};
}

uint64_t early_pairs(uint64_t cap, uint32_t probed) {
    return std::min(cap, std::min<uint64_t>(EARLY_PAIRS, std::max<uint64_t>(2048, probed / 16)));
}

uint64_t early_pairs(const JoinParams& P) {  // (a join of exchanged roles has no probe range)
    return early_pairs(P.out.cap, P.out.swap ? P.R.n : P.p_hi - P.p_lo);
}

hyset_status enqueue_result(hyset_ctx* ctx, const Sink& out, uint64_t early, const hyset_join_opts* o,
                            const PairSortJob* sort) {
    cudaStream_t s = ctx->stream;
    if (sort && !o->count_only && o->sort_pairs) CK(sort_pairs_cluster(*sort, s));
    CK(cudaMemcpyAsync(ctx->h_flags + 16, out.count, 8, cudaMemcpyDeviceToHost, s));
    if (!o->count_only && !o->device_pairs) {
        void* stage = nullptr;
        ST(host_stage(ctx, early * sizeof(hyset_pair), &stage));
        if (early) CK(cudaMemcpyAsync(stage, out.pairs, early * sizeof(hyset_pair), cudaMemcpyDeviceToHost, s));
    }
    return HYSET_OK;
}

hyset_status enqueue_result(hyset_ctx* ctx, const JoinParams& P, const hyset_join_opts* o) {
    const PairSortJob sort = pair_sort_job(P);
    return enqueue_result(ctx, P.out, early_pairs(P), o, &sort);
}

uint64_t joined_count(const hyset_ctx* ctx) {
    uint64_t count = 0;
    std::memcpy(&count, ctx->h_flags + 16, 8);
    return count;
}

hyset_status read_pairs(hyset_ctx* ctx, const void* d_pairs, uint64_t count, std::vector<hyset_pair>& out) {
    constexpr uint64_t STAGED_BYTES = 16ull << 20;  // larger results are copied straight to their place
    out.resize(count);
    if (count == 0) return HYSET_OK;
    const size_t bytes = count * sizeof(hyset_pair);
    void* to = out.data();
    if (bytes <= STAGED_BYTES) ST(host_stage(ctx, bytes, &to));
    CK(cudaMemcpyAsync(to, d_pairs, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (to != out.data()) std::memcpy(out.data(), to, bytes);
    return HYSET_OK;
}

hyset_status deliver_pairs(hyset_ctx* ctx, const JoinParams& P, const hyset_join_opts* o, hyset_result* res) {
    return deliver_pairs(ctx, early_pairs(P), P.out.swap ? P.R.n : P.S.n, P.out.swap ? P.S.n : P.R.n, o, res);
}

hyset_status deliver_pairs(hyset_ctx* ctx, uint64_t early, uint32_t n_probe, uint32_t n_indexed,
                           const hyset_join_opts* o, hyset_result* res) {
    if (o->count_only) return HYSET_OK;
    const bool resort = o->sort_pairs && res->count > PAIR_SORT_MAX;  // not sorted behind the join
    if (resort)
        ST(sort_device_pairs(ctx, ctx->s_pairs.as<uint2>(), res->count, n_probe, n_indexed));
    if (o->device_pairs) {
        if (resort) CK(cudaStreamSynchronize(ctx->stream));  // device pairs are final when the call returns
        res->device_pairs = ctx->s_pairs.p;
        return HYSET_OK;
    }
    if (!resort && res->count <= early) {  // all of them have come with their number
        const hyset_pair* staged = static_cast<const hyset_pair*>(ctx->h_stage);
        res->pairs.assign(staged, staged + res->count);
    } else {
        ST(read_pairs(ctx, ctx->s_pairs.p, res->count, res->pairs));
    }
    res->has_pairs = 1;
    return HYSET_OK;
}

hyset_status do_join(hyset_ctx* ctx, hyset_coll* R, hyset_coll* S, const hyset_join_opts* o, hyset_result* res) {
    ST(check_opts(ctx, o));
    const bool swapped = swap_sides(R, S, o);
    if (swapped) std::swap(R, S);
    const bool self = (S == R);
    if (self) {
        uint32_t split_at = 0;
        hyset_technique low = HYSET_TECH_AUTO, high = HYSET_TECH_AUTO;
        ST(plan_split(ctx, R, o, &split_at, &low, &high));
        if (split_at) {  // two probe ranges, each with its technique; pairs of the low range first
            hyset_result part[2];
            for (int k = 0; k < 2; ++k) {
                hyset_join_opts q = *o;
                q.technique = k == 0 ? low : high;
                q.probe_major = 1;
                q.probe_begin = k == 0 ? 0 : split_at;
                q.probe_end = k == 0 ? split_at : R->n;
                ST(do_join(ctx, R, S, &q, &part[k]));
            }
            res->count = part[0].count + part[1].count;
            res->has_pairs = part[0].has_pairs;
            res->pairs = std::move(part[0].pairs);
            res->pairs.insert(res->pairs.end(), part[1].pairs.begin(), part[1].pairs.end());
            res->device_ms = part[0].device_ms + part[1].device_ms;
            res->kernel_ms = part[0].kernel_ms + part[1].kernel_ms;
            for (int k = 0; k < 8; ++k) res->stats[k] = part[0].stats[k] + part[1].stats[k];
            res->launches = part[0].launches + part[1].launches;
            res->technique = part[1].technique;
            res->bitmap_bits = part[1].bitmap_bits;
            res->verify_mode = part[1].verify_mode;
            res->probe_batch = part[1].probe_batch;
            res->selector = 2;
            res->split_at = split_at;
            res->split_low = part[0].technique;
            return HYSET_OK;
        }
    }
    const uint32_t L = std::max(R->max_size, S->max_size);
    Bounds* b = nullptr;
    ST(get_bounds(ctx, o->sim, o->threshold, L, self ? 0 : 1, &b));
    hyset_technique selected = HYSET_TECH_AUTO;
    ST(select_technique(ctx, R, S, o, &selected, &res->selector));
    Tuned tn = tune(R, S, o, selected);
    const hyset_technique tech = tn.tech;
    res->technique = tech;
    {
        const uint32_t a_lo = o->probe_end ? o->probe_begin : 0, a_hi = o->probe_end ? o->probe_end : S->n;
        if (o->technique == HYSET_TECH_AUTO && o->bitmap_bits == 0 && tech == HYSET_TECH_FGSS && tn.probe_major &&
            a_hi - a_lo >= TUNE_MIN_PROBES)
            ST(autotune_bits(ctx, R, S, o, b, self, a_lo, a_hi, &tn.bits, o->verify_mode ? nullptr : &tn.vmode,
                             o->fgss_batch ? nullptr : &tn.batch));
    }
    const int vmode = tn.vmode;
    res->verify_mode = (uint32_t)vmode;
    res->bitmap_bits = tech == HYSET_TECH_DIRECT ? 0 : (tn.bits > 512 && !(tech == HYSET_TECH_FGSS && tn.probe_major) ? 512 : tn.bits);
    if (o->probe_end > S->n || o->probe_begin > o->probe_end)
        return fail(ctx, HYSET_E_INVALID, "probe range outside the probe collection");
    const unsigned long long launches0 = launches();
    CK(cudaEventRecord(ctx->ev0, ctx->stream));
    JoinParams P{};
    P.R = R->view();
    P.S = S->view();
    P.B = b->view;
    P.first_ge = R->first_ge.as<uint32_t>();
    P.R_L = R->max_size;
    P.self = self ? 1 : 0;
    P.grab = tech == HYSET_TECH_FGSS ? std::min<uint32_t>(tn.batch, 32) : 1;
    res->probe_batch = tech == HYSET_TECH_FGSS && tn.probe_major ? P.grab : 0;
    P.p_lo = o->probe_end ? o->probe_begin : 0;
    P.p_hi = o->probe_end ? o->probe_end : S->n;
    P.r_lo = 0;
    P.r_hi = R->n;
    P.out.swap = swapped ? 1 : 0;
    const bool token_major = tech == HYSET_TECH_FGSS && L < 65536 && !tn.probe_major;
    uint64_t group_entries = 0;
    TokenJoinParams T{};
    if (token_major) {
        // probes: maxprefix entries of S; candidates: the same groups (self-join,
        // midprefix filter in the kernel) or R's maxprefix entries (R-S join)
        const uint32_t U = std::max(R->universe, S->universe);
        ST(build_groups(ctx, S, b->view.probe_prefix, b->probe_prefix, U, &group_entries));
        if (!self) {
            uint64_t er = 0;
            ST(build_groups(ctx, R, b->view.index_prefix, b->index_prefix, U, &er));
            group_entries += er;
        }
        T.R = R->view();
        T.S = S->view();
        T.B = b->view;
        T.gs_off = S->g_off.as<uint32_t>();
        T.gs_set = S->g_set.as<uint32_t>();
        T.gs_ps = S->g_ps.as<uint32_t>();
        T.gr_off = R->g_off.as<uint32_t>();
        T.gr_set = R->g_set.as<uint32_t>();
        T.gr_ps = R->g_ps.as<uint32_t>();
        T.universe = U;
        T.self = self ? 1 : 0;
        T.grab = 16;
    }
    // signatures do not depend on the index: they are generated on the
    // auxiliary stream while the index builds on the context's stream
    // 1024-bit signatures serve the probe-major prefix filter; the window
    // techniques and the token-major kernel take 512 at most
    std::vector<JoinParams> parts;
    const int words = (int)(tn.bits / 64) > 8 && !(tech == HYSET_TECH_FGSS && tn.probe_major) ? 8 : (int)(tn.bits / 64);
    if (words) {
        const uint64_t *br = nullptr, *bs = nullptr;
        ST(get_bitmaps(ctx, R, words, &br, ctx->aux));
        if (self) bs = br;
        else ST(get_bitmaps(ctx, S, words, &bs, ctx->aux));
        P.bits_R = br;
        P.bits_S = bs;
        P.words = words;
        if (tech == HYSET_TECH_BITMAP) {
            split_window(R, S, b, words, P);
            if (!o->collect_stats) ST(widen_window(ctx, R, S, b, P, ctx->aux, parts));
        }
        CK(cudaEventRecord(ctx->ev_join, ctx->aux));
    }
    if (!token_major && tech == HYSET_TECH_FGSS) {
        ST(build_fgss_indexes(ctx, R, b, self, R->index, R->index_mid, P));
        if (P.X2.set) P.grab = std::min<uint32_t>(P.grab, 16);  // two bands per probe share a warp batch
        split_heavy(S, b, P);
    }
    if (words) CK(cudaStreamWaitEvent(ctx->stream, ctx->ev_join, 0));
    int ktech = tech == HYSET_TECH_FGSS ? TECH_FGSS : (tech == HYSET_TECH_DIRECT ? TECH_DIRECT : TECH_BITMAP);
    if (token_major) {
        T.bits_R = P.bits_R;
        T.bits_S = P.bits_S;
        T.words = P.words;
        if (o->probe_end && (o->probe_begin || o->probe_end != S->n))
            return fail(ctx, HYSET_E_UNSUPPORTED, "probe ranges need the probe-major kernel (probe_major = 1)");
        ST(run_join(ctx, P, ktech, vmode, o, res, true, &T));
        res->stats[3] = group_entries;
    } else {
        ST(run_join(ctx, P, ktech, vmode, o, res, true, nullptr, &parts));
    }
    if (P.X.set && o->collect_stats && !token_major) {
        res->stats[3] = R->index.entries;
    }
    res->launches = launches() - launches0;
    return HYSET_OK;
}

}  // namespace hs

using namespace hs;

extern "C" {

hyset_status hyset_self_join(hyset_ctx* ctx, const hyset_coll* coll, const hyset_join_opts* opts,
                             hyset_result** out) {
    if (!ctx || !coll || !out) return fail(ctx, HYSET_E_INVALID, "null argument");
    *out = nullptr;
    CK(cudaSetDevice(ctx->device));
    auto res = std::make_unique<hyset_result>();
    hyset_coll* c = const_cast<hyset_coll*>(coll);  // caches (index, signatures) live in the collection
    ST(do_join(ctx, c, c, opts, res.get()));
    *out = res.release();
    return HYSET_OK;
}

hyset_status hyset_rs_join(hyset_ctx* ctx, const hyset_coll* indexed, const hyset_coll* probe,
                           const hyset_join_opts* opts, hyset_result** out) {
    if (!ctx || !indexed || !probe || !out) return fail(ctx, HYSET_E_INVALID, "null argument");
    *out = nullptr;
    CK(cudaSetDevice(ctx->device));
    auto res = std::make_unique<hyset_result>();
    hyset_coll* R = const_cast<hyset_coll*>(indexed);
    hyset_coll* S = const_cast<hyset_coll*>(probe);
    if (R == S) return fail(ctx, HYSET_E_INVALID, "use hyset_self_join for R join R");
    ST(do_join(ctx, R, S, opts, res.get()));
    *out = res.release();
    return HYSET_OK;
}

}  // extern "C"
