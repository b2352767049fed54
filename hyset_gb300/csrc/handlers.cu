// handlers.cu — the reference-shaped handlers (bitmap::handler,
// fgssjoin::handler): block pairs and partitions of one collection, with the
// reference's per-indexed-block inverted index.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>

#include "host.h"

using namespace hs;

namespace {

// Room for `cap` pairs.  h->cap follows the buffer: a failed allocation leaves
// it at what the handler still holds (nothing, when the old buffer was given
// back for the new one), never at what was asked for.
cudaError_t pair_room(hyset_handler* h, uint64_t cap) {
    const cudaError_t e = h->pairs.ensure(cap * sizeof(uint2), h->ctx->stream);
    h->cap = e == cudaSuccess ? cap : std::min<uint64_t>(h->cap, h->pairs.bytes / sizeof(uint2));
    return e;
}

uint64_t least_pair_room(const hyset_handler* h) { return std::max<uint64_t>(1u << 16, (uint64_t)h->block_size * 4); }

}  // namespace

extern "C" {

hyset_status hyset_handler_create(hyset_ctx* ctx, const hyset_coll* coll, hyset_technique technique, hyset_sim sim,
                                  uint32_t bitmap_size, uint32_t block_size, int aggregate, double threshold,
                                  hyset_handler** out) {
    if (!ctx || !coll || !out) return fail(ctx, HYSET_E_INVALID, "null argument");
    *out = nullptr;
    if (technique != HYSET_TECH_BITMAP && technique != HYSET_TECH_FGSS)
        return fail(ctx, HYSET_E_INVALID, "handler technique must be BITMAP or FGSS");
    if (block_size == 0) return fail(ctx, HYSET_E_INVALID, "block size must be > 0");
    hyset_join_opts o;
    hyset_default_opts(&o);
    o.sim = sim;
    o.threshold = threshold;
    ST(check_opts(ctx, &o));
    if (technique == HYSET_TECH_BITMAP && bitmap_size != 64 && bitmap_size != 128 && bitmap_size != 256 &&
        bitmap_size != 512)
        return fail(ctx, HYSET_E_INVALID, "bitmap size must be 64, 128, 256 or 512");
    CK(cudaSetDevice(ctx->device));
    auto h = std::make_unique<hyset_handler>();
    auto guard = on_exit([&] {  // a failed creation releases what it allocated
        if (h) hyset_handler_destroy(h.release());
    });
    h->ctx = ctx;
    h->coll = coll;
    h->technique = technique;
    h->sim = sim;
    h->tau = threshold;
    h->block_size = block_size;
    h->aggregate = aggregate ? 1 : 0;
    ST(get_bounds(ctx, sim, threshold, coll->max_size, 0, &h->bounds));
    cudaStream_t s = ctx->stream;
    if (technique == HYSET_TECH_BITMAP) {
        // bitmap::handler ctor generates every signature up front (device_algorithms.hpp:144-156)
        h->words = (int)(bitmap_size / 64);
        CK(h->bits.ensure(sig_bytes(coll->n, h->words), s));
        CK(generate_signatures(coll, h->words, h->bits.as<uint64_t>(), s));
    }
    CK(h->count.ensure(16, s));
    CK(h->work.ensure(16, s));
    if (!h->aggregate) CK(pair_room(h.get(), least_pair_room(h.get())));
    CK(cudaStreamSynchronize(s));
    *out = h.release();
    return HYSET_OK;
}

namespace {

// Per-indexed-block inverted index in the reference's layout
// (include/hyset/index.hpp:284-313): zero universe-sized counts, histogram of
// the block's prefix entries, exclusive scan, atomic scatter (lists unsorted).
hyset_status build_block_index(hyset_handler* h, const hyset_block& blk) {
    hyset_ctx* ctx = h->ctx;
    cudaStream_t s = ctx->stream;
    const hyset_coll* c = h->coll;
    const uint32_t lo = blk.start_id, hi = blk.end_id + 1, nb = hi - lo, U = c->universe;
    uint64_t E = 0;  // the block's prefix entries (block.entries in the reference)
    const std::vector<uint64_t> bh = range_hist(c, lo, hi);
    for (size_t l = 0; l < bh.size(); ++l) E += bh[l] * h->bounds->index_prefix[l];
    const uint64_t E1 = E ? E : 1;
    h->indexed_block = -1;  // until the build is through: a failed one leaves no block's index
    CK(h->counts.ensure(((size_t)U + 1) * 4, s));
    CK(h->list_off.ensure(((size_t)U + 1) * 4, s));
    CK(h->e_len.ensure((size_t)nb * 4 + 4, s));
    CK(h->e_off.ensure((size_t)nb * 4 + 4, s));
    CK(h->e_tok.ensure(E1 * 4, s));
    CK(h->e_set.ensure(E1 * 4, s));
    CK(h->e_pos.ensure(E1 * 4, s));
    CK(h->idx_set.ensure(E1 * 4, s));
    CK(h->idx_pos.ensure(E1 * 4, s));
    CK(h->scan.ensure(std::max(scan_scratch_words(nb), scan_scratch_words((uint64_t)U + 1)) * 4, s));
    CollView v = c->view();
    uint32_t* scr = h->scan.as<uint32_t>();
    CK(set_prefix_lengths(v, h->bounds->view.index_prefix, lo, hi, h->e_len.as<uint32_t>(), s));
    CK(scan_exclusive(h->e_len.as<uint32_t>(), h->e_off.as<uint32_t>(), nb, scr, s));
    CK(emit_prefix_entries(v, lo, hi, h->e_off.as<uint32_t>(), h->e_len.as<uint32_t>(), h->e_tok.as<uint32_t>(),
                           h->e_set.as<uint32_t>(), h->e_pos.as<uint32_t>(), s));
    CK(cudaMemsetAsync(h->counts.p, 0, ((size_t)U + 1) * 4, s));
    CK(token_histogram(h->e_tok.as<uint32_t>(), E, h->counts.as<uint32_t>(), U + 1, s));
    CK(scan_exclusive(h->counts.as<uint32_t>(), h->list_off.as<uint32_t>(), (uint64_t)U + 1, scr, s));
    // the scatter advances a cursor copy of the list starts
    CK(cudaMemcpyAsync(h->counts.p, h->list_off.p, ((size_t)U + 1) * 4, cudaMemcpyDeviceToDevice, s));
    CK(scatter_entries(h->e_tok.as<uint32_t>(), h->e_set.as<uint32_t>(), h->e_pos.as<uint32_t>(), E,
                       h->counts.as<uint32_t>(), h->idx_set.as<uint32_t>(), h->idx_pos.as<uint32_t>(), s));
    h->indexed_block = blk.id;
    return HYSET_OK;
}

// One launch of the handler's technique, its pairs (or count) appended to the
// output; run again with room for everything when the pair buffer overflowed.
hyset_status run_handler_join(hyset_handler* h, JoinParams P) {
    hyset_ctx* ctx = h->ctx;
    cudaStream_t s = ctx->stream;
    if (!h->aggregate && h->cap == 0) CK(pair_room(h, least_pair_room(h)));  // lost to a failed allocation
    const int tech = h->technique == HYSET_TECH_FGSS ? TECH_FGSS : TECH_BITMAP;
    const int vmode = 1;
    hyset_join_opts o;
    hyset_default_opts(&o);
    o.count_only = (uint32_t)h->aggregate;
    for (int attempt = 0; attempt < 2; ++attempt) {
        P.out.pairs = h->aggregate ? nullptr : h->pairs.as<uint2>();
        P.out.count = h->count.as<unsigned long long>();
        P.out.cap = h->cap;
        P.out.count_only = h->aggregate;
        P.work = h->work.as<unsigned int>();
        CK(cudaMemsetAsync(h->count.p, 0, 16, s));
        CK(cudaMemsetAsync(h->work.p, 0, 16, s));
        CK(launch_join(P, tech, vmode, ctx->sm_count, s));
        ST(enqueue_result(ctx, P, &o));
        CK(cudaStreamSynchronize(s));
        const uint64_t count = joined_count(ctx);
        if (h->aggregate) {
            h->out_count += count;
            return HYSET_OK;
        }
        if (count <= h->cap) {
            if (count <= early_pairs(P)) {
                const hyset_pair* early = static_cast<const hyset_pair*>(ctx->h_stage);
                h->out_pairs.insert(h->out_pairs.end(), early, early + count);
            } else {
                std::vector<hyset_pair> got;
                ST(read_pairs(ctx, h->pairs.p, count, got));
                h->out_pairs.insert(h->out_pairs.end(), got.begin(), got.end());
            }
            h->out_count += count;
            return HYSET_OK;
        }
        CK(pair_room(h, count + count / 4 + 1024));
    }
    return fail(ctx, HYSET_E_OVERFLOW, "handler pair buffer overflow after resize");
}

hyset_status check_block(hyset_ctx* ctx, const hyset_coll* c, const hyset_block* b) {
    if (!b || b->start_id > b->end_id || b->end_id >= c->n) return fail(ctx, HYSET_E_INVALID, "bad block range");
    return HYSET_OK;
}

// A launch per block pair, each behind its own wait and each indexed block's
// lists built by ten kernels, made a partition join 272 launches for 20 blocks
// (4.05 ms for 200,000 short sets at Jaccard 0.8, half of it waiting).  Two
// runs of consecutive blocks are one join of two id ranges instead, with one
// sorted index of the indexed range, when the block pairs that the reference's
// id rule leaves out (probe block id below the indexed block's) hold no pair of
// a candidate before its probe; its length filter leaves out no pair of the
// result.  Blocks in another order, with gaps or with such ids go pair by pair,
// as do ranges of so many prefix entries that one index would take gigabytes,
// and ranges for whose index the device has no room.
bool joins_as_one(const hyset_handler* h, const hyset_block* first, uint32_t n_first, const hyset_block* second,
                  uint32_t n_second) {
    if (n_first == 0 || n_second == 0 || (uint64_t)n_first * n_second < 2) return false;
    const hyset_coll* c = h->coll;
    auto run = [c](const hyset_block* b, uint32_t n) {
        for (uint32_t i = 0; i < n; ++i)
            if (b[i].start_id > b[i].end_id || b[i].end_id >= c->n || (i && b[i].start_id != b[i - 1].end_id + 1))
                return false;
        return true;
    };
    if (!run(first, n_first) || !run(second, n_second)) return false;
    for (uint32_t i = 0; i < n_first; ++i)
        for (uint32_t k = 0; k < n_second; ++k)
            if (second[k].id < first[i].id && first[i].start_id < second[k].end_id) return false;
    constexpr uint64_t MOST_ENTRIES = 1ull << 28;  // about 8 GB of scratch
    return prefix_entries_of(range_hist(c, first[0].start_id, first[n_first - 1].end_id + 1),
                             h->bounds->index_prefix) < MOST_ENTRIES;
}

// Every pair of a probe in [p_lo, p_hi) and a candidate before it in [r_lo, r_hi).
hyset_status join_ranges(hyset_handler* h, uint32_t r_lo, uint32_t r_hi, uint32_t p_lo, uint32_t p_hi) {
    hyset_ctx* ctx = h->ctx;
    CK(cudaSetDevice(ctx->device));
    hyset_coll* c = const_cast<hyset_coll*>(h->coll);  // what it knows of its lists' lengths
    JoinParams P{};
    P.R = c->view();
    P.S = P.R;
    P.B = h->bounds->view;
    P.first_ge = c->first_ge.as<uint32_t>();
    P.R_L = c->max_size;
    P.self = 1;
    P.p_lo = p_lo;
    P.p_hi = p_hi;
    P.r_lo = r_lo;
    P.r_hi = r_hi;
    // room for a few pairs of every probe, as a whole join has (without it a
    // result that overflows is run again)
    const uint64_t room = std::min<uint64_t>(4ull * (p_hi - p_lo), 1u << 24);
    if (!h->aggregate && room > h->cap && pair_room(h, room) != cudaSuccess) (void)cudaGetLastError();
    if (h->technique == HYSET_TECH_FGSS) {
        P.grab = DEFAULT_PROBE_BATCH;
        ST(build_sorted_index(ctx, c, h->bounds, 0, h->part, nullptr, nullptr, -1, true, r_lo, r_hi));
        P.X = h->part.view();
        split_heavy(c, h->bounds, P);
    } else {
        P.grab = 1;
        P.bits_R = P.bits_S = h->bits.as<uint64_t>();
        P.words = h->words;
        split_window(c, c, h->bounds, h->words, P);
    }
    return run_handler_join(h, P);
}

}  // namespace

hyset_status hyset_handler_join_blocks(hyset_handler* h, const hyset_block* first, const hyset_block* second) {
    if (!h) return HYSET_E_INVALID;
    hyset_ctx* ctx = h->ctx;
    ST(check_block(ctx, h->coll, first));
    ST(check_block(ctx, h->coll, second));
    CK(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    if (h->technique == HYSET_TECH_FGSS && h->indexed_block != first->id) ST(build_block_index(h, *first));
    JoinParams P{};
    P.R = h->coll->view();
    P.S = P.R;
    P.B = h->bounds->view;
    P.first_ge = h->coll->first_ge.as<uint32_t>();
    P.R_L = h->coll->max_size;
    P.self = 1;
    P.grab = h->technique == HYSET_TECH_FGSS ? 4 : 1;
    P.p_lo = second->start_id;
    P.p_hi = second->end_id + 1;
    P.r_lo = first->start_id;
    P.r_hi = first->end_id + 1;
    if (h->technique == HYSET_TECH_FGSS) {
        P.X.list_off = h->list_off.as<uint32_t>();
        P.X.set = h->idx_set.as<uint32_t>();
        P.X.pos = h->idx_pos.as<uint32_t>();
        P.X.universe = h->coll->universe;
        P.X.sorted = 0;
    } else {
        P.bits_R = P.bits_S = h->bits.as<uint64_t>();
        P.words = h->words;
        split_window(h->coll, h->coll, h->bounds, h->words, P);
    }
    return run_handler_join(h, P);
}

hyset_status hyset_handler_join_partitions(hyset_handler* h, const hyset_block* first, uint32_t n_first,
                                           const hyset_block* second, uint32_t n_second) {
    if (!h || (n_first && !first) || (n_second && !second)) return HYSET_E_INVALID;
    if (joins_as_one(h, first, n_first, second, n_second)) {
        const hyset_status st = join_ranges(h, first[0].start_id, first[n_first - 1].end_id + 1, second[0].start_id,
                                            second[n_second - 1].end_id + 1);
        if (st != HYSET_E_NOMEM) return st;
        // nothing has come out yet: what the range's index took goes back, and one
        // block's index at a time does
        for (DevBuf* b : {&h->part.list_off, &h->part.set, &h->part.pos, &h->part.rec}) b->release(h->ctx->stream);
        h->ctx->sc->release(h->ctx->stream);
    }
    // device::length_filter (device_algorithms.hpp:21-53): probe block id >= indexed
    // block id and size[last indexed] >= minsize(size[first probe]).
    for (uint32_t i = 0; i < n_first; ++i) {
        ST(check_block(h->ctx, h->coll, &first[i]));
        for (uint32_t k = 0; k < n_second; ++k) {
            ST(check_block(h->ctx, h->coll, &second[k]));
            if (second[k].id < first[i].id) continue;
            uint32_t last_indexed = size_at(h->coll, first[i].end_id);
            uint32_t first_probe = size_at(h->coll, second[k].start_id);
            if (last_indexed >= h->bounds->minsize[first_probe]) ST(hyset_handler_join_blocks(h, &first[i], &second[k]));
        }
    }
    return HYSET_OK;
}

hyset_status hyset_handler_output(const hyset_handler* h, uint64_t* count, const hyset_pair** pairs) {
    if (!h) return HYSET_E_INVALID;
    if (count) *count = h->out_count;
    if (pairs) *pairs = h->aggregate ? nullptr : h->out_pairs.data();
    return HYSET_OK;
}

hyset_status hyset_handler_clear_output(hyset_handler* h) {
    if (!h) return HYSET_E_INVALID;
    h->out_count = 0;
    h->out_pairs.clear();
    return HYSET_OK;
}

void hyset_handler_destroy(hyset_handler* h) {
    if (!h) return;
    cudaStream_t s = h->ctx->stream;
    DevBuf* bufs[] = {&h->counts, &h->list_off, &h->e_len, &h->e_off, &h->e_tok, &h->e_set, &h->e_pos,
                      &h->idx_set, &h->idx_pos, &h->scan, &h->bits, &h->pairs, &h->count, &h->work,
                      &h->part.list_off, &h->part.set, &h->part.pos, &h->part.rec};
    for (DevBuf* b : bufs) b->release(s);
    cudaStreamSynchronize(s);
    delete h;
}

}  // extern "C"
