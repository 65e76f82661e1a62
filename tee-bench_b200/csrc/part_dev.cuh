// Device building blocks of the chunked radix partitioning (warp ranking,
// the TMA-fed digit-sorting tile scatter), shared by the single-join passes
// (partition.cu) and the batched join (batch.cu).
#pragma once

#include "tbg_device.cuh"

namespace tbg {

// ---------------------------------------------------------------------------
// shared helpers
// ---------------------------------------------------------------------------

// True when at least four neighbouring lane pairs of the warp hold the same
// digit: a sign of skew, for which the hot values' rows are aggregated (see
// hot_peers).  Fewer repeats (uniform keys over 128-256 digits give a pair
// in about one warp in five) cost less as plain atomics.
__device__ __forceinline__ bool warp_has_dups(uint32_t d, bool valid) {
    const int lane = threadIdx.x & 31;
    const uint32_t key = valid ? d : 0xFFFFFFFFu;
    const uint32_t up = __shfl_up_sync(0xffffffffu, key, 1);
    return __popc(__ballot_sync(0xffffffffu, valid && lane > 0 && up == key)) >= 4;
}

// Under skew a warp holds a few hot values among many distinct ones.  The
// lanes equal to lane 0's or lane 16's value (the likely hot ones) form a
// group: returns its lane mask for this lane, or 0 if this lane is in
// neither group.  Two shuffles and two ballots, whatever the spread.
__device__ __forceinline__ unsigned hot_peers(uint32_t key) {
    const uint32_t c0 = __shfl_sync(0xffffffffu, key, 0);
    const uint32_t c1 = __shfl_sync(0xffffffffu, key, 16);
    const unsigned g0 = __ballot_sync(0xffffffffu, key == c0);
    const unsigned g1 = __ballot_sync(0xffffffffu, key == c1 && key != c0);
    return key == c0 ? g0 : (key == c1 ? g1 : 0u);
}

// Adds one row's bin to a shared histogram; every lane of the warp calls it
// (valid = false for lanes without a row).  With `dup` (the warp showed
// repeated bins: skew), the hot groups add once per group; other rows pay
// one shared atomic each.
__device__ __forceinline__ void hist_add_warp(uint32_t *h, uint32_t f, bool valid, bool dup) {
    if (!dup) {
        if (valid) atomicAdd(&h[f], 1u);
    } else {
        const unsigned peers = hot_peers(valid ? f : 0xFFFFFFFFu);
        if (!valid) return;
        if (!peers) atomicAdd(&h[f], 1u);
        else if ((peers & lanemask_lt()) == 0) atomicAdd(&h[f], (uint32_t)__popc(peers));
    }
}

// Rank of a row on a shared digit counter (returns the old count).
// Correct either way; `dup` only picks the faster path.
__device__ __forceinline__ uint32_t rank_warp(uint32_t *cnt, uint32_t d, bool valid, bool dup) {
    uint32_t r = 0;
    if (!dup) {
        if (valid) r = atomicAdd(&cnt[d], 1u);
    } else {
        const unsigned peers = hot_peers(valid ? d : 0xFFFFFFFFu);
        const int leader = peers ? __ffs(peers) - 1 : 0;
        uint32_t b = 0;
        if (valid) {
            if (!peers) r = atomicAdd(&cnt[d], 1u);
            else if ((int)(threadIdx.x & 31) == leader) b = atomicAdd(&cnt[d], (uint32_t)__popc(peers));
        }
        // every lane joins both shuffles; group members take their leader's base
        const uint32_t b0 = __shfl_sync(0xffffffffu, b, leader);
        if (valid && peers) r = b0 + __popc(peers & lanemask_lt());
    }
    return r;
}

// ---------------------------------------------------------------------------
// tile scatter shared by both passes
// ---------------------------------------------------------------------------
// The elements of a pass: rows, or (counting joins, which need no payloads)
// bare keys.  A pass may read rows and write keys.
__device__ __forceinline__ uint32_t part_key(const Row &r) { return r.key; }
__device__ __forceinline__ uint32_t part_key(uint32_t k) { return k; }
__device__ __forceinline__ void part_conv(const Row &r, Row &o) { o = r; }
__device__ __forceinline__ void part_conv(const Row &r, uint32_t &o) { o = r.key; }
__device__ __forceinline__ void part_conv(uint32_t k, uint32_t &o) { o = k; }

// Tile buffers per CTA (the default): tile q is loaded and ranked while tile
// q - 1 is written out and tile q + 1 is being copied in.
constexpr int PART_NBUF = 3;

// A third barrier at the end of every tile (the layout before the tile loop
// was shown not to need it; kept as a build option for A/B timing).
#ifndef TBG_TILE_END_BARRIER
#define TBG_TILE_END_BARRIER 0
#endif

template <int THREADS, int NBUF = PART_NBUF, class In_ = Row, int ITEMS_ = PART_ITEMS>
struct PartSmem {
    using In = In_;
    static constexpr int NB = NBUF, ITEMS = ITEMS_;
    static constexpr int T = THREADS * ITEMS;
    static constexpr int VEC = 16 / sizeof(In);           // elements per 16 bytes
    In buf[NBUF][T + (2 * (VEC - 1) + VEC - 1) / VEC * VEC];  // input tiles (bulk copies), each then staged digit-sorted in place
    alignas(16) uint32_t cnt[2][SCATTER_FMAX];  // per-digit counts, then tile offsets, of the two newest tiles
    alignas(16) uint32_t delta[2][SCATTER_FMAX];  // output row - tile slot per digit, of the two newest tiles
    alignas(16) uint32_t cursor[SCATTER_FMAX];  // next output row of each digit
    uint64_t mbar[NBUF];
};

// Digit of a pass: a bit field of the key (pass 1: bits [0, b1); pass 2:
// bits [b1, b1 + b2); one pass: bits [0, B)).

// Destination shard of a key for a join split over n shards (n <= 256): the
// top bits of a multiplicative hash, range-reduced by a multiply-shift, so
// every shard gets an even share of the keys whatever their order or skew,
// and the low key bits that the shards' own radix passes use stay evenly
// spread inside each shard.
struct ShardOp {
    uint32_t n;
    __host__ __device__ __forceinline__ uint32_t operator()(uint32_t key) const {
        return (uint32_t)(((uint64_t)(key * 0x9E3779B1u) * n) >> 32);
    }
};

// Where tile elements [t, t + cnt) of an n-element array sit in a shared
// buffer: the bulk copy moves elements [t + c_lo, t + c_hi), a 16-byte aligned
// span; element r (relative to t) is at buffer index r + off, so the copy's
// destination is 16-byte aligned too.  When the tile starts or ends off a
// 16-byte boundary, the copy takes the neighbouring elements of the array as
// well, so the whole tile arrives by the bulk copy; only at the array's own
// ends, where there are not enough neighbours, are edge elements left out of
// the copy (those outside [a_lo, a_hi)) and read from global memory.
struct TileGeo {
    uint64_t t;
    uint32_t cnt, a_lo, a_hi, off;
    int32_t c_lo, c_hi;
};

template <class In>
__device__ __forceinline__ TileGeo tile_geo(const In *in, uint64_t t, uint32_t cnt, uint64_t n) {
    constexpr uint32_t VEC = 16 / sizeof(In);
    TileGeo g;
    g.t = t;
    g.cnt = cnt;
    const uintptr_t addr = reinterpret_cast<uintptr_t>(in + t);
    if constexpr (VEC == 2) {
        const bool lo_mis = (addr & 15) != 0;
        const bool hi_mis = ((addr + (uintptr_t)cnt * 8) & 15) != 0;
        g.c_lo = lo_mis ? (t >= 1 ? -1 : 1) : 0;
        g.c_hi = hi_mis ? (t + cnt < n ? (int32_t)cnt + 1 : (int32_t)cnt - 1) : (int32_t)cnt;
        g.off = lo_mis ? 1u : 0u;
    } else {
        const uint32_t lo_mis = (uint32_t)(addr & 15) / sizeof(In);
        const uint32_t hi_mis = (uint32_t)((addr + (uintptr_t)cnt * sizeof(In)) & 15) / sizeof(In);
        g.c_lo = lo_mis ? (t >= lo_mis ? -(int32_t)lo_mis : (int32_t)(VEC - lo_mis)) : 0;
        g.c_hi = hi_mis ? (t + cnt + (VEC - hi_mis) <= n ? (int32_t)(cnt + VEC - hi_mis) : (int32_t)cnt - (int32_t)hi_mis)
                        : (int32_t)cnt;
        g.off = lo_mis;
    }
    if (g.c_hi < g.c_lo) g.c_hi = g.c_lo;  // a few elements at an array end: no copy
    g.a_lo = (uint32_t)max(g.c_lo, 0);
    g.a_hi = (uint32_t)(VEC == 2 ? min(g.c_hi, (int32_t)cnt) : max(min(g.c_hi, (int32_t)cnt), 0));  // pairs: c_hi >= 0
    if (g.a_hi < g.a_lo) g.a_hi = g.a_lo;
    return g;
}

template <class In>
__device__ __forceinline__ void issue_tile(const In *in, const TileGeo &g, In *buf, uint64_t *bar) {
    const uint32_t bytes = (uint32_t)(g.c_hi - g.c_lo) * (uint32_t)sizeof(In);
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(bar, bytes);
    if (bytes) bulk_g2s(buf + g.c_lo + (int32_t)g.off, in + (int64_t)g.t + g.c_lo, bytes, bar);
}

// A tile's elements are read from its landed buffer and ranked on one shared
// counter per digit (order inside a digit is free: partitions are
// multisets); one warp prefixes the counts over digits while the other warps
// write out the previous tile; then the tile is staged digit-sorted into its
// own buffer, to be written out in slot order (consecutive threads store
// consecutive elements of each digit's run) during the next tile's prefix.
//
// Tile q (the CTA's running tile count, continued across ranges so a
// persistent CTA never re-initialises its barriers) uses buffer q % NB with
// barrier mbar[q % NB] at phase parity (q / NB) & 1, and counters and deltas
// q & 1.

// Waits for tile q and ranks its elements on cnt[q & 1].
template <bool FULL, class Out, class Dig, class Smem>
__device__ __forceinline__ void tile_load_rank(const typename Smem::In *__restrict__ in, const TileGeo &g, uint32_t q,
                                               Dig dop, Smem &sm, uint64_t *mbar, Out (&v)[Smem::ITEMS],
                                               uint32_t (&rank)[Smem::ITEMS], unsigned *err) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t wbase = (uint32_t)w * 32 * Smem::ITEMS;
    const uint32_t cnt = g.cnt;
    const int b = q % Smem::NB;
    if (!mbar_wait(&mbar[b], (q / Smem::NB) & 1, SPIN_LIMIT * 16)) atomicCAS(err, 0u, (unsigned)TBG_ERR_TIMEOUT);
#pragma unroll
    for (int i = 0; i < Smem::ITEMS; i++) {
        const uint32_t r = wbase + i * 32 + lane;
        if (FULL || r < cnt) {
            if (r >= g.a_lo && r < g.a_hi) part_conv(sm.buf[b][r + g.off], v[i]);
            else part_conv(in[g.t + r], v[i]);
        }
    }
    uint32_t *c = sm.cnt[q & 1];
    const bool dup = warp_has_dups(dop(part_key(v[0])), FULL || wbase + lane < cnt);
#pragma unroll
    for (int i = 0; i < Smem::ITEMS; i++) {
        const bool valid = FULL || wbase + i * 32 + lane < cnt;
        rank[i] = rank_warp(c, valid ? dop(part_key(v[i])) : 0, valid, dup);
    }
}

// Warp 0: digit counts of tile q -> tile offsets (in place), deltas and
// cursors; clears the counters of tile q + 1.  The tile lays the digits out
// in natural order, so neighbouring runs belong to neighbouring digits and a
// warp of the write-out that spans a run boundary reads its deltas from
// different banks.  Lane l owns the 8 consecutive digits [8l, 8l + 8) and
// moves them with 16-byte accesses (conflict-free).  Every counter of all
// SCATTER_FMAX digits is kept at zero outside the digits in use, so those
// add nothing.
template <class Smem>
__device__ __forceinline__ void tile_scan(uint32_t q, Smem &sm) {
    const int lane = threadIdx.x & 31;
    constexpr int PER = SCATTER_FMAX / 32;
    static_assert(PER == 8, "two 16-byte words of counters per lane");
    uint4 *c4 = reinterpret_cast<uint4 *>(sm.cnt[q & 1]) + 2 * lane;
    uint4 *d4 = reinterpret_cast<uint4 *>(sm.delta[q & 1]) + 2 * lane;
    uint4 *u4 = reinterpret_cast<uint4 *>(sm.cursor) + 2 * lane;
    uint4 *n4 = reinterpret_cast<uint4 *>(sm.cnt[(q + 1) & 1]) + 2 * lane;
    const uint4 ca = c4[0], cb = c4[1];
    const uint32_t x[PER] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < PER; i++) sum += x[i];
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    uint32_t run = inc - sum;
    const uint4 ua = u4[0], ub = u4[1];
    uint32_t cur[PER] = {ua.x, ua.y, ua.z, ua.w, ub.x, ub.y, ub.z, ub.w};
    uint32_t off[PER], dl[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) {
        off[i] = run;
        run += x[i];
        dl[i] = cur[i] - off[i];
        cur[i] += x[i];
    }
    c4[0] = make_uint4(off[0], off[1], off[2], off[3]);
    c4[1] = make_uint4(off[4], off[5], off[6], off[7]);
    d4[0] = make_uint4(dl[0], dl[1], dl[2], dl[3]);
    d4[1] = make_uint4(dl[4], dl[5], dl[6], dl[7]);
    u4[0] = make_uint4(cur[0], cur[1], cur[2], cur[3]);
    u4[1] = make_uint4(cur[4], cur[5], cur[6], cur[7]);
    n4[0] = make_uint4(0, 0, 0, 0);
    n4[1] = make_uint4(0, 0, 0, 0);
}

// Stages tile q's elements digit-sorted into its own buffer.
template <bool FULL, class Out, class Dig, class Smem>
__device__ __forceinline__ void tile_stage(const TileGeo &g, uint32_t q, Dig dop, Smem &sm, const Out (&v)[Smem::ITEMS],
                                           const uint32_t (&rank)[Smem::ITEMS]) {
    static_assert(sizeof(Out) <= sizeof(typename Smem::In), "staged in place");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t wbase = (uint32_t)w * 32 * Smem::ITEMS;
    const uint32_t *c = sm.cnt[q & 1];
    Out *buf = reinterpret_cast<Out *>(sm.buf[q % Smem::NB]);
#pragma unroll
    for (int i = 0; i < Smem::ITEMS; i++)
        if (FULL || wbase + i * 32 + lane < g.cnt) buf[c[dop(part_key(v[i]))] + rank[i]] = v[i];
}

// Writes staged tile q (cnt elements) to out, by threads [t0, THREADS).
template <int THREADS, class Out, class Dig, class Smem>
__device__ __forceinline__ void tile_write(uint32_t q, uint32_t cnt, Out *__restrict__ out, uint32_t out_n, Dig dop,
                                           Smem &sm, int t0, unsigned *err) {
    if ((int)threadIdx.x < t0) return;
    const Out *buf = reinterpret_cast<const Out *>(sm.buf[q % Smem::NB]);
    const uint32_t *dl = sm.delta[q & 1];
#pragma unroll 4
    for (uint32_t j = threadIdx.x - t0; j < cnt; j += THREADS - t0) {
        const Out x = buf[j];
        const uint32_t pos = dl[dop(part_key(x))] + j;
        if (pos < out_n) out[pos] = x;
        else atomicCAS(err, 0u, (unsigned)TBG_ERR_ARG);
    }
}

template <class In>
__device__ __forceinline__ TileGeo range_tile(const In *in, uint64_t lo, uint64_t hi, uint64_t n, int k, uint32_t T) {
    const uint64_t t = lo + (uint64_t)k * T;
    return tile_geo(in, t, (uint32_t)umin64(T, hi - t), n);
}

// Scatters elements [lo, hi) of `in` (in_n elements), digit by digit, to
// out[sm.cursor[d]...]; the caller initialises sm.cursor[0..F) and
// synchronises.  Two barriers per tile; the bulk copies run NB - 1 tiles
// ahead.  `kseq` is the CTA's running tile count (see above), and the barriers
// mbar[0..NB) are initialised once by the caller.
template <int THREADS, class Out, class Dig, class Smem>
__device__ void part_tiles(const typename Smem::In *__restrict__ in, uint64_t lo, uint64_t hi, uint64_t in_n,
                           Out *__restrict__ out, uint32_t out_n, Dig dop, Smem &sm, uint64_t *mbar, uint32_t &kseq,
                           unsigned *err) {
    constexpr uint32_t T = Smem::T;
    constexpr int NB = Smem::NB;
    const int ntiles = (int)((hi - lo + T - 1) / T);
    for (int i = threadIdx.x; i < SCATTER_FMAX; i += THREADS) sm.cnt[kseq & 1][i] = 0;
    __syncthreads();
    if (ntiles == 0) return;
    if (threadIdx.x == 0)
        for (int i = 0; i < NB - 1 && i < ntiles; i++)
            issue_tile(in, range_tile(in, lo, hi, in_n, i, T), sm.buf[(kseq + i) % NB], &mbar[(kseq + i) % NB]);
    uint32_t prev_cnt = 0;
    for (int k = 0; k < ntiles; k++) {
        const uint32_t q = kseq + k;
        const TileGeo g = range_tile(in, lo, hi, in_n, k, T);
        Out v[Smem::ITEMS];
        uint32_t rank[Smem::ITEMS];
        if (g.cnt == T) tile_load_rank<true, Out>(in, g, q, dop, sm, mbar, v, rank, err);
        else tile_load_rank<false, Out>(in, g, q, dop, sm, mbar, v, rank, err);
        __syncthreads();
        if (threadIdx.x < 32) tile_scan(q, sm);
        else if (k > 0) tile_write<THREADS, Out>(q - 1, prev_cnt, out, out_n, dop, sm, 32, err);
        __syncthreads();
        // tile q - 1's buffer is free: copy tile k + NB - 1 into it
        if (threadIdx.x == 0 && k + NB - 1 < ntiles)
            issue_tile(in, range_tile(in, lo, hi, in_n, k + NB - 1, T), sm.buf[(q + NB - 1) % NB],
                       &mbar[(q + NB - 1) % NB]);
        if (g.cnt == T) tile_stage<true, Out>(g, q, dop, sm, v, rank);
        else tile_stage<false, Out>(g, q, dop, sm, v, rank);
        // No barrier here: tile q + 1's load and ranking touch neither tile
        // q's buffer nor its counters, and the next iteration's first barrier
        // orders this staging before tile q's write-out and before the scan
        // that clears cnt[q & 1].
        if (TBG_TILE_END_BARRIER) __syncthreads();
        prev_cnt = g.cnt;
    }
    __syncthreads();  // the last tile is staged
    tile_write<THREADS, Out>(kseq + ntiles - 1, prev_cnt, out, out_n, dop, sm, 0, err);
    __syncthreads();  // every buffer is free again
    kseq += ntiles;
}

// One range per CTA: initialises the barriers held in `sm`.
template <int THREADS, class Out, class Dig, class Smem>
__device__ void part_range(const typename Smem::In *__restrict__ in, uint64_t lo, uint64_t hi, uint64_t in_n,
                           Out *__restrict__ out, uint32_t out_n, Dig dop, Smem &sm, unsigned *err) {
    if (threadIdx.x == 0) {
        for (int i = 0; i < Smem::NB; i++) mbar_init(&sm.mbar[i], 1);
        fence_mbar_init();
    }
    uint32_t kseq = 0;
    part_tiles<THREADS, Out>(in, lo, hi, in_n, out, out_n, dop, sm, sm.mbar, kseq, err);
}

}  // namespace tbg
