// Host pipelines of the sort-merge joins RSM and PSM.
//
// RSM (Joins/radix_sortmerge_join.c:102-105) shares RHO's radix partitioning
// and swaps the build/probe kernel for a per-partition sort + merge-path join.
// PSM (Joins/psm/parallel_sortmerge_join.h:61-111) sorts both relations by key
// and merges them.  The sort is MSD: RHO's histogram and passes partition by
// the top bits of key - min (at most 15), then every bucket is sorted by the
// remaining 12 or 13 bits in one counting pass (counting joins: every bucket's
// R rows are counted per key value, k_bucket_count).  Relations whose key range
// leaves more low bits, or with a bucket over a million rows (a heavy key),
// take an LSD radix sort (7- to 9-bit digits, chunked stable passes).
#include <algorithm>
#include <cstring>
#include <vector>

#include "tbg_internal.h"
#include "tbg_runtime.h"

namespace tbg {

cudaError_t launch_join_rsm(const JoinArgs &a, bool materialize, int grid, cudaStream_t st);
cudaError_t launch_merge_join(const Row *R, uint64_t nr, const Row *S, uint64_t ns, uint64_t *splits,
                              unsigned long long *matches, unsigned long long *rows_ctr, tbg_row_out *out,
                              uint64_t cap, bool mat, cudaStream_t st);
uint64_t merge_ctas(uint64_t nr, uint64_t ns);

constexpr int RSM_CAPR = 4096;

static void mark_ev(Workspace &w, bool timing, int i, cudaStream_t st) {
    if (timing) cudaEventRecord(w.ev[i], st);
}

int run_sortmerge_join(const tbg_config &cfg, const Row *dR, uint64_t nR, const Row *dS, uint64_t nS,
                       tbg_row_out *d_rows, uint64_t cap, Workspace &w, cudaStream_t st, JoinRun *run) {
    // one shared-memory radix-sorted tile (512 threads x 8 rows) of R per item
    const int capR = RSM_CAPR;
    if (nR <= SMALL_R) {
        const RadixGeom g = radix_geometry(cfg, nR, nS, capR, w);
        if (is_small_join(cfg, g)) return run_small_join(cfg, g, dR, dS, d_rows, cap, w, st, run);
    }
    int join_grid = 0;
    int rc = radix_partition(cfg, dR, nR, dS, nS, d_rows, cap, capR, w, st, run, &join_grid);
    if (rc) return rc;
    Ctrl *ctrl = w.ctrl.as<Ctrl>();
    JoinArgs ja;
    memset(&ja, 0, sizeof ja);
    ja.R = w.partR.as<Row>();
    ja.S = w.partS.as<Row>();
    ja.items = w.items.as<Item>();
    ja.nitems = &ctrl->nitems;
    ja.item_ctr = &ctrl->item_ctr[0];
    ja.capR = capR;
    ja.hash_shift = run->B;
    ja.matches = &ctrl->matches;
    ja.rows_ctr = &ctrl->rows;
    ja.out = d_rows;
    ja.cap = d_rows ? cap : 0;
    ja.err = &ctrl->error;
    ja.skip = &ctrl->direct;
    cudaError_t e =
        launch_join_rsm(ja, cfg.materialize != 0, w.nsm * rsm_ctas_per_sm(capR, cfg.materialize != 0), st);
    if (e != cudaSuccess) return cuda_error(e, "rsm join");
    mark_ev(w, cfg.timing != 0, 4, st);
    run->timed = cfg.timing != 0;
    return TBG_OK;
}

cudaError_t launch_sort_pass(const Row *in, Row *out, uint64_t n, uint64_t chunk, int G, const uint32_t *pre,
                             const uint32_t *totals, uint32_t shift, uint32_t sub, int digit_bits, unsigned *err,
                             cudaStream_t st);

// Passes of the LSD sort of keys in [kmin, kmax]: (shift, digit bits) over
// the bits of key - kmin, the fewest passes of at most 9 bits with the bits
// spread evenly (at least 7 per pass: at an equal pass count narrower digits
// are cheaper to rank and give longer runs per digit).  Sorting by key - kmin
// keeps the key order and needs only the bits of the range: 3 passes for
// the keys 1..2^27 (27 bits of range), where the raw keys span 28 bits.
std::vector<std::pair<uint32_t, int>> sort_plan(uint32_t kmin, uint32_t kmax) {
    std::vector<std::pair<uint32_t, int>> plan;
    if (kmax <= kmin) return plan;
    const uint32_t span = kmax - kmin;
    const int bits = 32 - __builtin_clz(span);
    const int np = (bits + 8) / 9;
    const int db = std::max(7, (bits + np - 1) / np);
    for (int i = 0, lo = 0; i < np; i++, lo += db) plan.push_back({(uint32_t)lo, std::min(db, 32 - lo)});
    return plan;
}

// LSD sort of n rows by key with chunked stable passes (per-chunk digit
// histograms, column prefix, k_sort_pass): 24 B per row per pass and no
// inter-CTA waits.  Digits are taken from key - kmin.
int lsd_sort_chunked(const Row *in, uint64_t n, uint32_t kmin, uint32_t kmax, DevBuf &a, DevBuf &b, Workspace &w,
                     cudaStream_t st, const Row **out, int *passes) {
    const Row *src = in;
    Row *bufs[2] = {a.as<Row>(), b.as<Row>()};
    int which = 0;
    *passes = 0;
    const int G = (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)w.nsm * 4, (n + 32767) / 32768));
    const uint64_t chunk = (n + G - 1) / G;
    cudaError_t e = w.sorthist.ensure(((size_t)G + 1) * 512 * 4);
    if (e != cudaSuccess) return cuda_error(e, "cudaMalloc");
    uint32_t *hist = w.sorthist.as<uint32_t>(), *totals = hist + (size_t)G * 512;
    unsigned *err = &w.ctrl.as<Ctrl>()->error;
    if (n <= 1) {
        *out = src;
        return TBG_OK;
    }
    for (const auto &pp : sort_plan(kmin, kmax)) {
        const uint32_t shift = pp.first;
        const int db = pp.second;
        const uint32_t m2 = (1u << db) - 1;
        RadixF rf{0u, shift, m2, 0u};
        rf.sub = kmin;
        if ((e = launch_hist_chunks(src, n, chunk, G, hist, db, rf, st)) != cudaSuccess ||
            (e = launch_colscan(hist, G, 1 << db, totals, st)) != cudaSuccess ||
            (e = launch_sort_pass(src, bufs[which], n, chunk, G, hist, totals, shift, kmin, db, err, st)) !=
                cudaSuccess)
            return cuda_error(e, "sort pass");
        src = bufs[which];
        which ^= 1;
        (*passes)++;
    }
    *out = src;
    return TBG_OK;
}

cudaError_t launch_bucket_sort(const Row *in, Row *out, const uint64_t *base, uint32_t nb, uint64_t n, uint32_t sub,
                               int lowbits, int nsm, cudaStream_t st);

// MSD sort of both relations: radix partitioning by the top B bits of
// key - sub (RHO's histogram and passes), then each bucket sorted by the low
// `lowbits` bits (k_bucket_sort), into sorted[0] (R) and sorted[1] (S).  A
// relation with a bucket over kBucketMax rows (a heavy key) is left for the
// LSD sort instead: msd_done[rel] says which ones were sorted.
static constexpr uint64_t kBucketMax = 1u << 20;
static constexpr int kLowBits = 12, kLowBitsMax = 13;

// Radix bits and low bits of an MSD sort of keys that span `span` bits; false
// when the LSD sort takes them (no bits above the low ones, or too many low
// bits).
static bool msd_bits(int span, int *B, int *lowbits) {
    *lowbits = std::min(span, kLowBits);
    *B = span - *lowbits;
    if (*B > 15) {
        *B = 15;
        *lowbits = span - *B;
    }
    return *B >= 1 && *lowbits <= kLowBitsMax;
}

uint64_t heavy_bucket_rows(uint64_t nR, int nsm);
cudaError_t launch_bucket_count(const JoinArgs &a, const HeavyBuckets &hv, uint32_t sub, int lowbits, int nsm,
                                cudaStream_t st);

// Count-only PSM on MSD buckets: both relations partitioned by the top bits of
// key - sub (sub, rmax: R's key range), then k_bucket_count.  Nothing waits, and
// neither S's keys outside R's range nor heavy keys (S's buckets are split over
// CTAs by the planner, R's rows of a large bucket counted once) need another
// plan.
// lsd_passes > 0: the range has no bits above the low ones, where the sort
// would be an LSD sort of that many passes; the buckets do for it too.
static int msd_count(const tbg_config &cfg, const Row *dR, uint64_t nR, const Row *dS, uint64_t nS, uint32_t sub,
                     uint32_t rmax, int B, int lowbits, int lsd_passes, Workspace &w, cudaStream_t st, JoinRun *run) {
    if (lsd_passes) {  // a range of at most kLowBits bits: two buckets
        B = 1;
        lowbits = std::max(lowbits - 1, 2);
    }
    // one radix bit less where both plans take two passes: a pass costs more
    // per bit above 7 than the larger buckets do (8 + 7 bits against 7 + 7 at
    // 2^27 x 2^30: 4.64 against 3.79 ms for the second pass)
    if (B > 9 && lowbits < kLowBitsMax) {
        B--;
        lowbits++;
    }
    RadixGeom g = radix_geometry_msd(nR, nS, sub, B, lowbits, w);
    try_direct(g, cfg, nullptr, 0);
    if (nR > (uint64_t)(rmax - sub) + 1) g.direct = false;  // more rows than key values: not distinct
    g.sample_S = dS;
    g.capR = 0x7FFFFFFF;  // counters take any number of R rows
    g.keys = true;
    g.split.rows = g.split.wide = std::max<uint64_t>(65536, nS / ((uint64_t)w.nsm * 12));
    g.item_cap = 2 * (nS / g.split.rows + 4 * g.P) + 16;
    int rc = ensure_radix_buffers(g, false, w);
    if (rc) return rc;
    if ((rc = start_radix_join(g, dR, w, st)) || (rc = part_hist_read(0, g, dR, cfg, w, st, nullptr)) || (rc = part_hist_read(1, g, dS, cfg, w, st, nullptr)) ||
        (rc = part_hist_plan(3, true, g, w, st)) || (rc = both_passes(cfg, g, dR, dS, w, st)))
        return rc;
    Ctrl *ctrl = w.ctrl.as<Ctrl>();
    JoinArgs ja;
    memset(&ja, 0, sizeof ja);
    ja.R = w.partR.as<Row>();
    ja.S = w.partS.as<Row>();
    ja.items = w.items.as<Item>();
    ja.nitems = &ctrl->nitems;
    ja.item_ctr = &ctrl->item_ctr[0];
    ja.matches = &ctrl->matches;
    ja.err = &ctrl->error;
    ja.skip = &ctrl->direct;
    HeavyBuckets hv;
    hv.rows = heavy_bucket_rows(nR, w.nsm);
    if (nR <= hv.rows) {
        hv.rows = 0;  // no bucket can be
    } else if (w.aux[5].ensure(((nR / hv.rows + 1) << lowbits) * 4) != cudaSuccess) {
        cudaGetLastError();
        hv.rows = 0;  // no memory for the counters: every item counts its bucket's rows
    }
    hv.nR = nR;
    hv.counters = w.aux[5].as<uint32_t>();
    hv.base = w.baseR.as<uint64_t>();
    hv.max_part = &ctrl->max_part_R;
    const cudaError_t e = launch_bucket_count(ja, hv, sub, lowbits, w.nsm, st);
    if (e != cudaSuccess) return cuda_error(e, "bucket count");
    mark_ev(w, cfg.timing != 0, 4, st);
    run->B = lsd_passes ? 8 : B;
    run->passes = lsd_passes ? lsd_passes : g.passes + 1;  // the count takes the place of the bucket sort
    run->P = lsd_passes ? 0 : g.P;
    run->timed = cfg.timing != 0;
    return TBG_OK;
}

// With check_s, the range [sub, sub + 2^span) is R's alone: S's histogram
// also counts S's keys outside it, and if there are any, nothing is sorted
// and *s_outside is set (the caller then takes both relations' range).
// The first sort (check_s) also tries the direct join during the histogram
// reads: with *direct set the join is done.
static int msd_sort(const tbg_config &cfg, const Row *dR, uint64_t nR, const Row *dS, uint64_t nS, uint32_t sub,
                    int span, bool check_s, tbg_row_out *d_rows, uint64_t cap, Row *sorted[2], bool msd_done[2],
                    bool *s_outside, bool *direct, Workspace &w, cudaStream_t st, JoinRun *run) {
    msd_done[0] = msd_done[1] = false;
    *s_outside = *direct = false;
    int B, lowbits;
    if (!msd_bits(span, &B, &lowbits)) return TBG_OK;  // the LSD sort takes both
    RadixGeom g = radix_geometry_msd(nR, nS, sub, B, lowbits, w);
    if (check_s) g.s_range_max = (uint32_t)((1ull << span) - 1);
    if (check_s) try_direct(g, cfg, d_rows, cap);
    int rc = ensure_radix_buffers(g, false, w);
    if (rc) return rc;
    Ctrl *ctrl = w.ctrl.as<Ctrl>();
    cudaError_t e;
    if ((rc = start_radix_join(g, dR, w, st))) return rc;
    if ((rc = part_hist_read(0, g, dR, cfg, w, st, nullptr)) || (rc = part_hist_read(1, g, dS, cfg, w, st, nullptr)) ||
        (rc = part_hist_plan(3, false, g, w, st)))
        return rc;
    // the largest bucket of each relation decides between this sort and LSD;
    // S's keys outside R's range void the histograms
    if ((e = cudaMemcpyAsync(w.host_ctrl, ctrl, sizeof(Ctrl), cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return cuda_error(e, "bucket sizes");
    const Ctrl &hc = *w.host_ctrl;
    if (!hc.direct && check_s && hc.out_of_range) {
        *s_outside = true;
        return TBG_OK;
    }
    run->B = B;
    run->passes = g.passes + 1;
    run->P = g.P;
    if (hc.direct) {
        *direct = true;
        return TBG_OK;
    }
    const unsigned long long maxp[2] = {hc.max_part_R, hc.max_part_S};
    const Row *in[2] = {dR, dS};
    for (int rel = 0; rel < 2; rel++) {
        if (maxp[rel] > kBucketMax) continue;
        if ((rc = part_pass(rel, 1, g, in[rel], w, st, false)) || (rc = part_pass(rel, 2, g, in[rel], w, st, false)))
            return rc;
        const Row *part = (rel ? w.partS : w.partR).as<Row>();
        const uint64_t *base = (rel ? w.baseS : w.baseR).as<uint64_t>();
        if ((e = launch_bucket_sort(part, sorted[rel], base, (uint32_t)g.P, rel ? nS : nR, sub, lowbits, w.nsm,
                                    st)) != cudaSuccess)
            return cuda_error(e, "bucket sort");
        msd_done[rel] = true;
        mark_ev(w, cfg.timing != 0, 2 + rel, st);
    }
    return TBG_OK;
}

// The direct join in front of the LSD sort (key ranges without MSD buckets,
// when R's range fits the table): its histograms have two bins, only to be
// thrown away.  *direct: the join is done.
static int direct_or_lsd(const tbg_config &cfg, const Row *dR, uint64_t nR, const Row *dS, uint64_t nS, uint32_t rmin,
                         uint32_t rmax, tbg_row_out *d_rows, uint64_t cap, bool *direct, Workspace &w, cudaStream_t st) {
    *direct = false;
    RadixGeom g = radix_geometry_msd(nR, nS, rmin, 1, 31, w);
    try_direct(g, cfg, d_rows, cap);
    g.sample_S = dS;
    const int lg = g.direct_rows ? direct_log2_max_rows(nR) : direct_log2_max(nR);
    // more rows than key values: not distinct
    if (!g.direct || (uint64_t)(rmax - rmin) >= (1ull << lg) || nR > (uint64_t)(rmax - rmin) + 1) return TBG_OK;
    cudaError_t e;
    if ((e = w.histR.ensure((uint64_t)g.G[0] * g.P * 4)) != cudaSuccess ||
        (e = w.histS.ensure((uint64_t)g.G[1] * g.P * 4)) != cudaSuccess)
        return cuda_error(e, "cudaMalloc");
    int rc;
    if ((rc = start_radix_join(g, dR, w, st)) || (rc = part_hist_read(0, g, dR, cfg, w, st, nullptr)) ||
        (rc = part_hist_read(1, g, dS, cfg, w, st, nullptr)))
        return rc;
    if ((e = cudaMemcpyAsync(w.host_ctrl, w.ctrl.p, sizeof(Ctrl), cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return cuda_error(e, "direct join");
    *direct = w.host_ctrl->direct != 0;
    return TBG_OK;
}

int run_psm_join(const tbg_config &cfg, const Row *dR, uint64_t nR, const Row *dS, uint64_t nS,
                 tbg_row_out *d_rows, uint64_t cap, Workspace &w, cudaStream_t st, JoinRun *run) {
    const bool timing = cfg.timing != 0;
    cudaError_t e;
#define ENSURE(buf, bytes)                                        \
    do {                                                          \
        e = (buf).ensure(bytes);                                  \
        if (e != cudaSuccess) return cuda_error(e, "cudaMalloc"); \
    } while (0)
    ENSURE(w.ctrl, sizeof(Ctrl));
    ENSURE(w.aux[4], 64);
    Ctrl *ctrl = w.ctrl.as<Ctrl>();
    uint32_t *mm = w.aux[4].as<uint32_t>();  // min, max of R's keys, then of S's
    uint32_t *hm = static_cast<uint32_t *>(w.host_small);
    mark_ev(w, timing, 0, st);
    if ((e = cudaMemsetAsync(ctrl, 0, sizeof(Ctrl), st)) != cudaSuccess) return cuda_error(e, "memset");
    // R's key range decides the MSD geometry (S's keys usually lie inside it:
    // S's histogram checks that, so S's own range read is only needed when
    // they do not, or for the LSD sort)
    uint32_t rmin = 0, rmax = 0, smin = 0, smax = 0;
    bool have_s = false;
    auto read_range = [&](const Row *d, uint64_t n, uint32_t *lo, uint32_t *hi) -> int {
        if ((e = launch_key_range(d, n, mm, w.nsm, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(hm, mm, 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
            (e = cudaStreamSynchronize(st)) != cudaSuccess)
            return cuda_error(e, "key range");
        *lo = hm[0];
        *hi = hm[1];
        return TBG_OK;
    };
    auto span_of = [](uint32_t lo, uint32_t hi) { return hi > lo ? 32 - __builtin_clz(hi - lo) : 0; };
    int rc = read_range(dR, nR, &rmin, &rmax);
    if (rc) return rc;
    mark_ev(w, timing, 1, st);
    int B = 0, lowbits = 0;
    if (!cfg.materialize && nR && nS) {
        if (msd_bits(span_of(rmin, rmax), &B, &lowbits))
            return msd_count(cfg, dR, nR, dS, nS, rmin, rmax, B, lowbits, 0, w, st, run);
        if (span_of(rmin, rmax) <= kLowBits)
            return msd_count(cfg, dR, nR, dS, nS, rmin, rmax, 1, lowbits,
                             std::max<int>(1, (int)sort_plan(rmin, rmax).size()), w, st, run);
    }
    bool direct = false;
    run->B = 8;
    run->P = 0;
    run->passes = 0;
    auto done_direct = [&]() -> int {
        for (int i = 2; i <= 4; i++) mark_ev(w, timing, i, st);
        run->timed = timing;
        return TBG_OK;
    };
    if (nR && nS && !msd_bits(span_of(rmin, rmax), &B, &lowbits)) {
        if ((rc = direct_or_lsd(cfg, dR, nR, dS, nS, rmin, rmax, d_rows, cap, &direct, w, st))) return rc;
        if (direct) {
            run->passes = (int)sort_plan(rmin, rmax).size();
            return done_direct();
        }
    }
    ENSURE(w.aux[0], nR * 8);
    ENSURE(w.aux[1], nR * 8);
    ENSURE(w.aux[2], nS * 8);
    ENSURE(w.aux[3], nS * 8);
    ENSURE(w.aux[6], (merge_ctas(nR, nS) + 2) * 8);
#undef ENSURE
    Row *sorted[2] = {w.aux[0].as<Row>(), w.aux[2].as<Row>()};
    bool msd_done[2] = {false, false};
    if (nR && nS) {
        bool s_outside = false;
        if ((rc = msd_sort(cfg, dR, nR, dS, nS, rmin, span_of(rmin, rmax), true, d_rows, cap, sorted, msd_done, &s_outside,
                           &direct, w, st, run)))
            return rc;
        if (direct) return done_direct();
        if (s_outside) {  // both relations' range, histograms again
            if ((rc = read_range(dS, nS, &smin, &smax))) return rc;
            have_s = true;
            const uint32_t lo = std::min(rmin, smin), hi = std::max(rmax, smax);
            if ((rc = msd_sort(cfg, dR, nR, dS, nS, lo, span_of(lo, hi), false, d_rows, cap, sorted, msd_done, &s_outside,
                               &direct, w, st, run)))
                return rc;
        }
    }
    const Row *sR = sorted[0], *sS = sorted[1];
    int pr = 0, ps = 0;
    if (!msd_done[0]) {
        if ((rc = lsd_sort_chunked(dR, nR, rmin, rmax, w.aux[0], w.aux[1], w, st, &sR, &pr))) return rc;
        mark_ev(w, timing, 2, st);
    }
    if (!msd_done[1]) {
        if (!have_s && (rc = read_range(dS, nS, &smin, &smax))) return rc;
        if ((rc = lsd_sort_chunked(dS, nS, smin, smax, w.aux[2], w.aux[3], w, st, &sS, &ps))) return rc;
        mark_ev(w, timing, 3, st);
    }
    e = launch_merge_join(sR, nR, sS, nS, w.aux[6].as<uint64_t>(), &ctrl->matches, &ctrl->rows, d_rows,
                          d_rows ? cap : 0, cfg.materialize != 0, st);
    if (e != cudaSuccess) return cuda_error(e, "merge join");
    mark_ev(w, timing, 4, st);
    if (!msd_done[0] || !msd_done[1]) run->passes = std::max(run->passes, std::max(pr, ps));
    run->timed = timing;
    return TBG_OK;
}

}  // namespace tbg
