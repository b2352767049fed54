// index_host.cu — host orchestration of the index builds: size statistics of
// a collection, the global set-id-sorted prefix index (and the R-S midprefix
// index), token groups, and the XOR signatures.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>

#include "host.h"

namespace hs {

// Host size statistics from host-resident sizes (the caller's array, or the
// pinned copy of device sizes): the per-size histogram and first_ge[l] = first
// set id with size >= l (sizes are non-decreasing), whose device copy is
// enqueued on the stream (the host array is a member, so no synchronisation is
// needed here).  The collection keeps no per-set host array: sizes of single
// sets and of id ranges come from first_ge.
namespace {
// first_ge (and its device copy) and the largest size from the histogram.
hyset_status finish_size_meta(hyset_ctx* ctx, hyset_coll* c) {
    const uint32_t L = (uint32_t)c->size_hist.size() - 1;
    c->max_size = L;
    std::vector<uint32_t>& f = c->h_first_ge;
    f.resize((size_t)L + 2);
    uint64_t run = 0;
    for (uint32_t l = 0; l <= L + 1; ++l) {
        f[l] = (uint32_t)run;
        if (l <= L) run += c->size_hist[l];
    }
    CK(c->first_ge.ensure(f.size() * 4, ctx->stream));
    CK(cudaMemcpyAsync(c->first_ge.p, f.data(), f.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
    return HYSET_OK;
}
}  // namespace

hyset_status build_size_meta(hyset_ctx* ctx, hyset_coll* c, const uint32_t* sizes) {
    std::vector<uint64_t>& hist = c->size_hist;
    hist.assign(c->n ? (size_t)sizes[c->n - 1] + 1 : 1, 0);
    uint32_t i = 0;
    // run lengths: sorted sizes repeat, so the count stays in a register
    while (i < c->n) {
        const uint32_t v = sizes[i];
        uint32_t j = i + 1;
        while (j < c->n && sizes[j] == v) ++j;
        if (v >= hist.size()) hist.resize((size_t)v + 1, 0);
        hist[v] += j - i;
        i = j;
    }
    return finish_size_meta(ctx, c);
}

hyset_status build_size_meta_runs(hyset_ctx* ctx, hyset_coll* c, const uint32_t* runs, uint32_t n_runs) {
    std::vector<std::pair<uint32_t, uint32_t>> by(n_runs);  // (first set, size): sizes are non-decreasing
    for (uint32_t k = 0; k < n_runs; ++k) by[k] = {runs[2 * k + 1], runs[2 * k]};
    std::sort(by.begin(), by.end());
    c->size_hist.assign(n_runs ? (size_t)by.back().second + 1 : 1, 0);
    for (uint32_t k = 0; k < n_runs; ++k)
        c->size_hist[by[k].second] += (k + 1 < n_runs ? by[k + 1].first : c->n) - by[k].first;
    return finish_size_meta(ctx, c);
}

void size_meta_from_first_ge(hyset_coll* c, const uint32_t* first_ge, uint32_t L) {
    c->max_size = L;
    c->h_first_ge.assign(first_ge, first_ge + (size_t)L + 2);
    c->size_hist.assign((size_t)L + 1, 0);
    for (uint32_t l = 0; l <= L; ++l) c->size_hist[l] = first_ge[l + 1] - first_ge[l];
}

// Size of set i (sizes are non-decreasing: the last l with first_ge[l] <= i).
uint32_t size_at(const hyset_coll* c, uint32_t i) {
    const auto& f = c->h_first_ge;
    return (uint32_t)(std::upper_bound(f.begin(), f.end(), i) - f.begin()) - 1;
}

// Sets per size among ids [lo, hi).
std::vector<uint64_t> range_hist(const hyset_coll* c, uint32_t lo, uint32_t hi) {
    std::vector<uint64_t> ph((size_t)c->max_size + 1, 0);
    const auto& f = c->h_first_ge;
    for (uint32_t l = 0; l <= c->max_size; ++l) {
        const uint32_t a = std::max(lo, f[l]), b = std::min(hi, f[l + 1]);
        if (b > a) ph[l] = b - a;
    }
    return ph;
}

// Prefix entries of sets [lo, hi) (all sets when hi == n) from the size histogram.
uint64_t prefix_entries(const hyset_coll* c, const std::vector<uint32_t>& pre) {
    uint64_t E = 0;
    for (size_t l = 0; l < c->size_hist.size(); ++l) E += c->size_hist[l] * (uint64_t)pre[l];
    return E;
}

uint64_t prefix_entries_of(const std::vector<uint64_t>& hist, const std::vector<uint32_t>& pre) {
    uint64_t E = 0;
    for (size_t l = 0; l < hist.size(); ++l) E += hist[l] * (uint64_t)pre[l];
    return E;
}

BoundFields bound_fields(const Bounds* b) {
    return BoundFields{b->view.max_sum, b->view.lp_row, b->view.lp_tab};
}

uint32_t first_long_prefix(const hyset_coll* c, const std::vector<uint32_t>& pre) {
    constexpr uint32_t LONG_PREFIX = 32;  // longer prefixes are emitted a warp per set
    uint64_t id = 0;
    for (size_t l = 0; l < c->size_hist.size(); ++l) {
        if (l < pre.size() && pre[l] > LONG_PREFIX) return (uint32_t)id;
        id += c->size_hist[l];
    }
    return 0xFFFFFFFFu;
}

void entry_layout(const hyset_coll* c, const Bounds* b, int kind, uint32_t pb, uint32_t* low_bits, bool* bound) {
    const uint32_t fb = bits_for(b->L);  // a field that holds every probe length
    *bound = kind == 0 && (b->view.max_sum != nullptr || b->view.lp_tab != nullptr) && fb + bits_for(c->n) <= 32;
    *low_bits = *bound ? fb : pb;
}

// Bits needed to represent v (at least 1).
uint32_t bits_for(uint64_t v) {
    uint32_t b = 1;
    while (b < 64 && (v >> b)) ++b;
    return b;
}


int key_bits_for(uint32_t universe) {
    int bits = 1;
    while (bits < 32 && (universe - 1) >> bits) ++bits;
    return bits;
}

// Global inverted index over the prefix entries of every set, lists ordered by
// set id: histogram + scan give the list offsets; the entries (emitted in set
// order) go into their lists by atomic slots and each list is put back in set
// order in shared memory when every list is short, or by a stable radix sort
// by token otherwise (index_lists).
// pre / d_pre: the prefix length table (default: the bounds' index prefix);
// force_pb >= 0 fixes the layout (0 = unpacked, > 0 = packed with that many
// position bits) so that two indexes of one join share it.
// records_ok: the caller's kernel reads token records (record_shift); they are
// built where the longest list of this prefix table fits (it is read back on
// the collection's first build with the table, which guesses the width) and
// there is room for them, directly from the prefix entries: one emit pass and
// one ordering pass, no offsets, no scan.
// [lo, hi): only these sets are indexed (set ids stay absolute).
hyset_status build_sorted_index(hyset_ctx* ctx, hyset_coll* c, const Bounds* b, int kind, Index& ix,
                                const std::vector<uint32_t>* pre, const uint32_t* d_pre,
                                int force_pb, bool records_ok, uint32_t lo, uint32_t hi) {
    // Rebuilt on every join (buffers are reused): a join's timed device work
    // always includes its own index build.  Only asynchronous stream work once
    // the buffers are large enough, so a batch can capture it into a graph.
    if (!pre) {
        pre = &b->index_prefix;
        d_pre = b->view.index_prefix;
    }
    cudaStream_t s = ctx->stream;
    const uint32_t n = c->n, U = c->universe;
    hi = std::min(hi, n);
    const bool whole = lo == 0 && hi == n;
    const uint64_t E = whole ? prefix_entries(c, *pre) : prefix_entries_of(range_hist(c, lo, hi), *pre);
    if (E >= (1ull << 32)) return fail(ctx, HYSET_E_UNSUPPORTED, "more than 2^32 prefix entries");
    const uint64_t E1 = E ? E : 1;
    CK(ctx->sc->len.ensure((size_t)n * 4 + 4, s));
    CK(ctx->sc->off.ensure((size_t)n * 4 + 4, s));
    CK(ctx->sc->tok.ensure(E1 * 4, s));
    CK(ctx->sc->set.ensure(E1 * 4, s));
    CK(ctx->sc->pos.ensure(E1 * 4, s));
    CK(ctx->sc->order.ensure(E1 * 4, s));
    CK(ctx->sc->altk.ensure(E1 * 4, s));
    CK(ctx->sc->altv.ensure(E1 * 4, s));
    CK(ctx->sc->counts.ensure(((size_t)U + 1) * 4, s));
    size_t scan_words = std::max(std::max(scan_scratch_words(n), scan_scratch_words((uint64_t)U + 1)),
                                 radix_scratch_words(E1));
    CK(ctx->sc->scan.ensure(scan_words * 4, s));
    CK(ix.list_off.ensure(((size_t)U + 1) * 4, s));
    CK(ix.set.ensure(E1 * 4, s));
    CK(ix.pos.ensure(E1 * 4, s));
    CollView v = c->view();
    uint32_t* len = ctx->sc->len.as<uint32_t>();
    uint32_t* off = ctx->sc->off.as<uint32_t>();
    uint32_t* scr = ctx->sc->scan.as<uint32_t>();
    // Packed entries (set << pb | position) when set ids up to n and positions
    // below the longest prefix fit 32 bits: the sorted values are the index.
    uint32_t max_pre = 1;
    for (size_t l = 0; l < c->size_hist.size(); ++l)
        if (c->size_hist[l]) max_pre = std::max(max_pre, (*pre)[l]);
    const uint32_t pb = force_pb > 0 ? (uint32_t)force_pb : bits_for(max_pre), sb = bits_for(n);
    const bool packed = force_pb != 0 && pb + sb <= 32;
    // Records are sized from the longest list seen on an earlier build, so only
    // collections whose tokens the library owns (immutable once uploaded) use
    // them; a collection over caller memory can change between joins.
    const bool owned = c->tokens.p != nullptr && c->d_tokens == c->tokens.as<uint32_t>();
    const bool rec_fits = records_ok && packed && owned;
    ix.sim = b->sim;
    ix.tau = b->tau;
    ix.kind = kind;
    ix.universe = U;
    ix.entries = E;
    ix.records = 0;
    ix.low_bits = packed ? pb : 0;
    ix.bound = false;
    // the kernel that reads records reads bound fields, in records or lists
    if (packed && records_ok) entry_layout(c, b, kind, pb, &ix.low_bits, &ix.bound);
    const BoundFields bf = ix.bound ? bound_fields(b) : BoundFields{};
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    CK(cudaStreamIsCapturing(s, &capture));
    const bool capturing = capture != cudaStreamCaptureStatusNone;
    // Room for records of this shift; without it the lists do.  (A capture
    // allocates nothing: its buffers were sized before it.)
    auto room = [&](int shift) {
        const size_t need = ((size_t)U << shift) * 4;
        if (capturing) return ix.rec.p && ix.rec.bytes >= need;
        if (ix.rec_guessed && ix.rec.bytes > need) ix.rec.release(s);  // wider than its lists turned out to need
        ix.rec_guessed = false;
        return ix.rec.ensure(need, s) == cudaSuccess;
    };
    auto emit_in_records = [&](int shift) -> hyset_status {
        CK(cudaMemsetAsync(ctx->sc->counts.p, 0, (size_t)U * 4, s));
        CK(emit_records(v, d_pre, ix.low_bits, ctx->sc->counts.as<uint32_t>(), ix.rec.as<uint32_t>(), shift, U, s, lo,
                        hi, bf, first_long_prefix(c, *pre)));
        return HYSET_OK;
    };
    auto finish_records = [&](int shift) -> hyset_status {
        CK(order_records(ctx->sc->counts.as<uint32_t>(), U, ix.rec.as<uint32_t>(), shift, s));
        ix.records = shift;
        ix.pos_bits = pb;
        return HYSET_OK;
    };
    if (rec_fits) {
        auto lk = c->list_longest.find(d_pre);
        // The first build with this prefix table does not know its longest list.
        // Where the average is short enough that it may fit, the entries go into
        // records at once and their counts are read back; lists, an offset scan,
        // a scatter, a ranking and a conversion took 90 us longer for 200,000
        // long sets.  Longer lists than a record holds are built again below.
        // Narrow records up to one entry per token on average: the first join of
        // 1,024 sets over 2^24 tokens takes 0.60 ms and 2.2 GB with them, 0.80 and
        // 4.4 with the wide ones, 1.36 and 2.2 by way of lists.
        constexpr uint64_t MAY_FIT = 16;  // entries per token: a longest list of 63 is four times this
        const int guess = E <= U ? 5 : E <= MAY_FIT * U ? 6 : 0;
        if (lk == c->list_longest.end() && whole && E && guess && record_shift(record_entries(guess), U) == guess &&
            !capturing && room(guess)) {
            CK(ctx->sc->gate.ensure(4, s));
            ST(emit_in_records(guess));
            int& path = c->list_path[d_pre];
            CK(longest_list(ctx->sc->counts.as<uint32_t>(), U, ctx->sc->gate.as<uint32_t>(), s, ctx->h_flags + 15, &path));
            lk = c->list_longest.emplace(d_pre, ctx->h_flags[15]).first;
            const int needs = record_shift(lk->second, U);
            if (needs && needs <= guess) {
                ix.rec_guessed = needs < guess;
                return finish_records(guess);
            }
            if (!needs) ix.rec.release(s);
        }
        const int shift = lk != c->list_longest.end() ? record_shift(lk->second, U) : 0;
        if (shift && room(shift)) {
            ST(emit_in_records(shift));
            return finish_records(shift);
        }
    }
    CK(set_prefix_lengths(v, d_pre, lo, hi, len + lo, s));  // len and off by absolute set id
    CK(scan_exclusive(len + lo, off + lo, hi - lo, scr, s));
    if (packed) {
        uint32_t* counts = ctx->sc->counts.as<uint32_t>();
        CK(ctx->sc->gate.ensure(4, s));
        CK(cudaMemsetAsync(counts, 0, ((size_t)U + 1) * 4, s));
        CK(emit_packed_entries(v, off, len, ix.low_bits, ctx->sc->tok.as<uint32_t>(), ix.set.as<uint32_t>(), counts, s,
                               lo, hi, 0xFFFFFFFFu, first_long_prefix(c, *pre), bf));
        // the list build's path is read back once per collection and prefix
        // table (not while a batch is being captured into a graph)
        // (a part of the collection has no longer lists than the whole, but says
        // nothing about it: its own path is not remembered)
        const auto known = c->list_path.find(d_pre);
        int part_path = known == c->list_path.end() ? 0 : known->second;
        int& path = whole ? c->list_path[d_pre] : part_path;
        const bool read_back = path == 0 && !capturing;
        CK(index_lists(ctx->sc->tok.as<uint32_t>(), ix.set.as<uint32_t>(), E, U, counts, ix.list_off.as<uint32_t>(),
                       ctx->sc->altk.as<uint32_t>(), ctx->sc->altv.as<uint32_t>(), ctx->sc->gate.as<uint32_t>(),
                       key_bits_for(U), scr, s, &path, read_back ? ctx->h_flags + 15 : nullptr));
        if (read_back && E && whole) c->list_longest[d_pre] = ctx->h_flags[15];
        ix.pos_bits = pb;
        const int shift = rec_fits && E && read_back ? record_shift(ctx->h_flags[15], U) : 0;
        if (shift && room(shift)) {
            // this build's lists become records; later builds emit records directly
            CK(records_from_lists(ix.list_off.as<uint32_t>(), ix.set.as<uint32_t>(), U, ix.rec.as<uint32_t>(), shift,
                                  s));
            ix.records = shift;
        }
        return HYSET_OK;
    }
    CK(emit_prefix_entries(v, lo, hi, off + lo, len + lo, ctx->sc->tok.as<uint32_t>(), ctx->sc->set.as<uint32_t>(),
                           ctx->sc->pos.as<uint32_t>(), s));
    uint32_t* counts = ctx->sc->counts.as<uint32_t>();
    CK(cudaMemsetAsync(counts, 0, ((size_t)U + 1) * 4, s));
    CK(token_histogram(ctx->sc->tok.as<uint32_t>(), E, counts, U + 1, s));
    CK(scan_exclusive(counts, ix.list_off.as<uint32_t>(), (uint64_t)U + 1, scr, s));
    CK(iota_u32(ctx->sc->order.as<uint32_t>(), E, s));
    CK(radix_sort_pairs(ctx->sc->tok.as<uint32_t>(), ctx->sc->order.as<uint32_t>(), ctx->sc->altk.as<uint32_t>(),
                        ctx->sc->altv.as<uint32_t>(), E, key_bits_for(U), scr, s, false));
    CK(gather_entries(ctx->sc->order.as<uint32_t>(), E, ctx->sc->set.as<uint32_t>(), ctx->sc->pos.as<uint32_t>(),
                      ix.set.as<uint32_t>(), ix.pos.as<uint32_t>(), s));
    ix.sim = b->sim;
    ix.tau = b->tau;
    ix.kind = kind;
    ix.universe = U;
    ix.entries = E;
    ix.pos_bits = 0;
    return HYSET_OK;
}

// R-S prefix-index joins split each probe's length window in two bands:
// candidates at least as long as the probe need only the probe's midprefix
// tokens (against R's maxprefix index), shorter candidates need only their
// own midprefix entries (a second, midprefix index of R, against the probe's
// maxprefix tokens).  Both hold because minoverlap does not decrease when
// either length grows, which get_bounds checks on the bound tables.
bool use_bands(const Bounds* b, bool self) { return !self && b->mo_monotone; }

// The prefix index (and for banded R-S joins the midprefix index) of R, and
// their views in P.
hyset_status build_fgss_indexes(hyset_ctx* ctx, hyset_coll* R, const Bounds* b, bool self, Index& ix,
                                 Index& ix_mid, JoinParams& P) {
    ST(build_sorted_index(ctx, R, b, self ? 0 : 1, ix, nullptr, nullptr, -1, true));
    P.X = ix.view();
    P.X2 = IndexView{};
    if (use_bands(b, self)) {
        ST(build_sorted_index(ctx, R, b, 2, ix_mid, &b->mid_prefix, b->view.mid_prefix, (int)ix.pos_bits, true));
        P.X2 = ix_mid.view();
    }
    return HYSET_OK;
}

// Token groups of the first pre[size] tokens of every set (histogram, scan,
// atomic scatter).  Rebuilt on every join; buffers are reused.
hyset_status build_groups(hyset_ctx* ctx, hyset_coll* c, const uint32_t* d_pre, const std::vector<uint32_t>& pre,
                          uint32_t U, uint64_t* entries) {
    cudaStream_t s = ctx->stream;
    const uint64_t E = prefix_entries(c, pre);
    if (E >= (1ull << 32)) return fail(ctx, HYSET_E_UNSUPPORTED, "more than 2^32 prefix entries");
    CK(c->g_off.ensure(((size_t)U + 1) * 4, s));
    CK(c->g_cursor.ensure(((size_t)U + 1) * 4, s));
    CK(c->g_set.ensure((E ? E : 1) * 4, s));
    CK(c->g_ps.ensure((E ? E : 1) * 4, s));
    CK(ctx->sc->scan.ensure(scan_scratch_words((uint64_t)U + 1) * 4, s));
    uint32_t* cnt = c->g_cursor.as<uint32_t>();
    CK(cudaMemsetAsync(cnt, 0, ((size_t)U + 1) * 4, s));
    CK(group_count(c->view(), d_pre, cnt, s));
    CK(scan_exclusive(cnt, c->g_off.as<uint32_t>(), (uint64_t)U + 1, ctx->sc->scan.as<uint32_t>(), s));
    CK(cudaMemcpyAsync(cnt, c->g_off.p, ((size_t)U + 1) * 4, cudaMemcpyDeviceToDevice, s));
    CK(group_scatter(c->view(), d_pre, cnt, c->g_set.as<uint32_t>(), c->g_ps.as<uint32_t>(), s));
    *entries = E;
    return HYSET_OK;
}

cudaError_t generate_signatures(const hyset_coll* c, int words, uint64_t* out, cudaStream_t s, unsigned max_blocks) {
    uint64_t long_tokens = 0;
    for (size_t l = SIG_WARP_SIZE; l < c->size_hist.size(); ++l) long_tokens += c->size_hist[l] * l;
    const uint32_t long_lo = c->max_size >= SIG_WARP_SIZE ? c->h_first_ge[SIG_WARP_SIZE] : c->n;
    return generate_bitmaps(c->view(), words, out, s, long_lo,
                            c->n_tokens ? (double)long_tokens / (double)c->n_tokens : 0.0, max_blocks);
}

// Signatures are regenerated on every join (the buffer is reused); the buffer
// is sized on the context's stream, the generation runs on `gen` (default: the
// same stream).
hyset_status get_bitmaps(hyset_ctx* ctx, hyset_coll* c, int words, const uint64_t** out,
                         cudaStream_t gen) {
    DevBuf& d = c->bitmaps[words];
    CK(d.ensure(sig_bytes(c->n, words), ctx->stream));
    if (gen && gen != ctx->stream) {
        CK(cudaEventRecord(ctx->ev_fork, ctx->stream));
        CK(cudaStreamWaitEvent(gen, ctx->ev_fork, 0));
    }
    // beside the index build the generation takes a few blocks per SM (it is
    // bandwidth-bound; the index build is latency-bound and needs the SMs)
    const unsigned cap = gen && gen != ctx->stream ? (unsigned)(ctx->sm_count * HS_SIG_BLOCKS_PER_SM) : 0u;
    CK(generate_signatures(c, words, d.as<uint64_t>(), gen ? gen : ctx->stream, cap));
    *out = d.as<uint64_t>();
    return HYSET_OK;
}

}  // namespace hs
