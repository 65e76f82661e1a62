// Device building blocks of the build/probe join (shared-memory bucket-chain
// or histogram table, count probe), shared by the single-join kernel
// (join.cu) and the batched join (batch.cu).
#pragma once

#include "tbg_device.cuh"

namespace tbg {

// Largest power of two <= x (x >= 1).
__host__ __device__ __forceinline__ uint32_t floor_pow2(uint32_t x) {
    uint32_t p = 1;
    while (p <= x / 2) p <<= 1;
    return p;
}

// Histogram-table probes read the bucket's keys four at a time (a build
// option for A/B timing).
#ifndef TBG_RHT_VEC_PROBE
#define TBG_RHT_VEC_PROBE 1
#endif

struct Table {
    uint32_t *key;    // [capR]
    uint32_t *pay;    // [capR]
    uint32_t *heads;  // layout 0: [N] 1-based chain heads; layout 1: [Nb+1] starts, then cursors
    uint16_t *next;   // layout 0: [capR] 1-based next links
    uint32_t mask;    // bucket mask
    uint32_t hcap;    // head slots available (a power of two <= capR + 2)
    int hs;           // hash shift (radix bits already consumed)
    int layout;

    __device__ __forceinline__ uint32_t bucket(uint32_t k) const { return (k >> hs) & mask; }

    template <class Fn>
    __device__ __forceinline__ void for_each(uint32_t k, Fn fn) const {
        const uint32_t b = bucket(k);
        if (layout == 0) {
            for (uint32_t h = heads[b]; h; h = next[h - 1])
                if (key[h - 1] == k) fn(pay[h - 1]);
        } else {
            for (uint32_t j = heads[b], e = heads[b + 1]; j < e; j++)
                if (key[j] == k) fn(pay[j]);
        }
    }
    __device__ __forceinline__ uint32_t count(uint32_t k) const {
        uint32_t c = 0;
        const uint32_t b = bucket(k);
        if (layout == 0) {
            for (uint32_t h = heads[b]; h; h = next[h - 1]) c += (key[h - 1] == k);
        } else if (TBG_RHT_VEC_PROBE) {
            // the bucket's keys read as 16-byte words (key[] starts 16-byte
            // aligned): a word's slots before the bucket hold keys of other
            // buckets, which differ from k; slots at or past its end are
            // masked (past the table they may hold stale keys)
            const uint32_t j = heads[b], e = heads[b + 1];
            const uint4 *k4 = reinterpret_cast<const uint4 *>(key);
            for (uint32_t a4 = j & ~3u; a4 < e; a4 += 4) {
                const uint4 q = k4[a4 >> 2];
                c += (q.x == k) + (q.y == k && a4 + 1 < e) + (q.z == k && a4 + 2 < e) + (q.w == k && a4 + 3 < e);
            }
        } else {
            for (uint32_t j = heads[b], e = heads[b + 1]; j < e; j++) c += (key[j] == k);
        }
        return c;
    }
};


// Long runs of one key in a table of R rows: the buckets with chains of
// RUN_ROWS cells or more, and how many rows each key in them has.  A lookup
// then reads one count where the chain costs a dependent load per row.
constexpr uint32_t RUN_ROWS = 128;  // a table of 16384 rows holds at most RUN_BUCKETS such runs
constexpr uint32_t RUN_BUCKETS = 128, RUN_KEYS = 256;
constexpr uint32_t RUN_NONE = 0xFFFFFFFFu;
struct LongRuns {
    uint32_t bucket[RUN_BUCKETS];       // hashed set, RUN_NONE: free
    uint32_t key[RUN_KEYS];             // hashed, RUN_NONE: free
    uint32_t rows[RUN_KEYS];            // R rows of the key
    uint32_t full;                      // no room: the chains stay

    __device__ __forceinline__ static uint32_t hash(uint32_t x, uint32_t n) { return (x * 0x9E3779B1u >> 16) & (n - 1); }
    // Slot of x in set[n], or (not there) the first free slot after its hash,
    // or n.
    __device__ __forceinline__ static uint32_t find(const uint32_t *set, uint32_t n, uint32_t x) {
        uint32_t h = hash(x, n);
        for (uint32_t t = 0; t < n; t++, h = (h + 1) & (n - 1))
            if (set[h] == x || set[h] == RUN_NONE) return h;
        return n;
    }
    // The same, entering x where it is not there.
    __device__ __forceinline__ static uint32_t enter(uint32_t *set, uint32_t n, uint32_t x) {
        uint32_t h = hash(x, n);
        for (uint32_t t = 0; t < n; t++, h = (h + 1) & (n - 1)) {
            const uint32_t seen = set[h] == x ? x : atomicCAS(&set[h], RUN_NONE, x);
            if (seen == RUN_NONE || seen == x) return h;
        }
        return n;
    }
    __device__ __forceinline__ uint32_t count(uint32_t k) const {
        const uint32_t h = find(key, RUN_KEYS, k);
        return h < RUN_KEYS && key[h] == k && k != RUN_NONE ? rows[h] : 0u;
    }
};

// Count-only bucket chains of 32-bit cells.  With q = key >> hs, row i's
// bucket is q mod N and its tag the bits of q above that, which with the
// bucket and the low hs bits (shared by all rows of the join's partition)
// make up the whole key: a cell needs no key beside it.  A cell holds {tag,
// link}, link the 1-based place in `cells` of the next cell of the chain (0:
// the end); a new row's cell becomes the bucket's head and the head it
// displaces moves to cells[i].  The tag has 32 - link_bits bits, so N is at
// least 2^(link_bits - hs).  Against 64-bit heads {key, row, link} with keys
// and links in arrays of their own (112 KB at 8192 rows, two CTAs per SM) a
// lookup reads one 4-byte word instead of 8 bytes, and 10240 rows take 72 KB,
// three CTAs per SM.
//
// With `runs` set, buckets with long chains are counted per key instead
// (LongRuns), and CELL_RUN is their head; has_runs says that there are any (the
// same for all threads), for which the probe has a loop of its own: the test in
// every lookup took 2% of a 16 M x 134 M join.  2^20 x 2^24 rows with 4096 rows
// a key take 0.20 ms, 46 ms along the chains; with 256 rows a key 0.19 and 3.0;
// with 1% of R on one key (2^20 x 2^22) 0.13 and 3.3, most of it the swaps in
// build_cells.  Counting RHO and RHT take it, the batch (whose plan has the
// histogram table to choose) does not.
constexpr uint32_t CELL_EMPTY = 0xFFFFFFFFu;  // the links of these two are past any row
constexpr uint32_t CELL_RUN = 0xFFFFFFFEu;

struct CellTable {
    uint32_t *heads;  // [N <= hcap]
    uint32_t *cells;  // [rows]
    uint32_t hcap;    // a power of two
    int hs, link_bits;
    uint32_t mask;    // N - 1
    int tag_shift;    // hs + log2 N
    LongRuns *runs = nullptr;
    bool has_runs = false;

    template <bool RUNS = false>
    __device__ __forceinline__ uint32_t count(uint32_t k) const {
        uint32_t c = heads[(k >> hs) & mask];
        if (c >= (RUNS ? CELL_RUN : CELL_EMPTY)) return RUNS && c == CELL_RUN ? runs->count(k) : 0u;
        const uint32_t tag = tag_shift < 32 ? k >> tag_shift : 0u;
        const uint32_t lmask = (1u << link_bits) - 1;
        uint32_t n = 0;
        for (;;) {
            n += (c >> link_bits) == tag;
            const uint32_t l = c & lmask;
            if (!l) return n;
            c = cells[l - 1];
        }
    }
};

// Link bits of a table of `rows` rows: links 0 .. rows, and two values more.
__host__ __device__ __forceinline__ int cell_link_bits(uint32_t rows) {
    int b = 1;
    while ((1u << b) < rows + 3) b++;
    return b;
}

// R rows are read with plain loads, or with L2-only loads (CG) when they were
// written earlier in the same kernel launch by other CTAs.
template <bool CG>
__device__ __forceinline__ uint2 ld_row(const Row *R, uint64_t i) {
    const uint2 *p = reinterpret_cast<const uint2 *>(R) + i;
    if (CG) return __ldcg(p);
    return *p;
}
template <bool CG>
__device__ __forceinline__ uint32_t ld_key(const Row *R, uint64_t i) { return ld_row<CG>(R, i).x; }
template <bool CG>
__device__ __forceinline__ uint32_t ld_key(const uint32_t *R, uint64_t i) { return CG ? __ldcg(R + i) : R[i]; }

// A row, or a bare key with no payload.
template <bool CG>
__device__ __forceinline__ uint2 ld_elem(const Row *R, uint64_t i) { return ld_row<CG>(R, i); }
template <bool CG>
__device__ __forceinline__ uint2 ld_elem(const uint32_t *R, uint64_t i) { return make_uint2(ld_key<CG>(R, i), 0u); }
template <bool CG>
__device__ __forceinline__ uint4 ld_pair(const uint4 *p) {
    if (CG) return __ldcg(p);
    return ldg_stream(p);
}

// Finds the long chains of a built table and counts their keys' rows (see
// LongRuns); true when there are any.  The caller has a barrier before, and
// this ends with one.  The first THREADS rows look along their chains: a run of
// RUN_ROWS among 10240 rows has one of 512 of them but once in 600 tables, and
// then stays a chain.
template <int THREADS, bool CG, class E>
__device__ __forceinline__ bool collapse_runs(uint32_t *heads, const uint32_t *cells, uint32_t mask, int hs, int link_bits,
                                           const E *__restrict__ R, uint32_t r_len, LongRuns *lr) {
    const uint32_t tid = threadIdx.x, lmask = (1u << link_bits) - 1;
    bool found = false;
    uint32_t b0 = 0;
    if (tid < r_len) {
        b0 = (ld_key<CG>(R, tid) >> hs) & mask;
        uint32_t n = 1;
        for (uint32_t c = heads[b0]; n < RUN_ROWS && (c & lmask); n++) c = cells[(c & lmask) - 1];
        found = n == RUN_ROWS;
    }
    if (!__syncthreads_or(found)) return false;
    for (uint32_t i = tid; i < RUN_KEYS; i += THREADS) {
        lr->key[i] = RUN_NONE;
        lr->rows[i] = 0;
        if (i < RUN_BUCKETS) lr->bucket[i] = RUN_NONE;
    }
    if (tid == 0) lr->full = 0;
    __syncthreads();
    if (found) LongRuns::enter(lr->bucket, RUN_BUCKETS, b0);
    __syncthreads();
    for (uint32_t i = tid; i < r_len; i += THREADS) {
        const uint32_t k = ld_key<CG>(R, i), b = (k >> hs) & mask;
        const uint32_t q = LongRuns::find(lr->bucket, RUN_BUCKETS, b);
        if (q == RUN_BUCKETS || lr->bucket[q] != b) continue;
        const uint32_t h = k == RUN_NONE ? RUN_KEYS : LongRuns::enter(lr->key, RUN_KEYS, k);
        if (h < RUN_KEYS) atomicAdd(&lr->rows[h], 1u);
        else lr->full = 1;
    }
    __syncthreads();
    if (lr->full) return false;
    if (tid < RUN_BUCKETS && lr->bucket[tid] != RUN_NONE) heads[lr->bucket[tid]] = CELL_RUN;
    __syncthreads();
    return true;
}

// The same as a function: k_join's probe keeps its registers. (The one-launch
// join has registers to spare, and a function cost it 0.2 of 26 us.)
template <int THREADS, bool CG, class E>
__device__ __noinline__ bool collapse_runs_call(uint32_t *heads, const uint32_t *cells, uint32_t mask, int hs, int link_bits,
                                                const E *__restrict__ R, uint32_t r_len, LongRuns *lr) {
    return collapse_runs<THREADS, CG>(heads, cells, mask, hs, link_bits, R, r_len, lr);
}
enum Runs { RUNS_NONE, RUNS_CALL, RUNS_INLINE };  // whether, and how, a build looks for long runs

// Builds the cells of R rows [r_off, r_off + r_len); ends with a barrier.  A
// row whose swap fails finds another row's cell at the head, never the empty
// one, so it exchanges its cell for whatever is there and does not try again
// (in a loop of swaps 10,000 rows of one key took 3 ms).
// RUNS: a row that displaces a cell of its own tag says that there may be long
// runs (or a key twice: a look at 512 chains finds those short).
template <int THREADS, bool CG = false, Runs RUNS = RUNS_NONE, class E = Row>
__device__ __forceinline__ void build_cells(CellTable &t, const E *__restrict__ R, uint64_t r_off, uint32_t r_len) {
    const int tid = threadIdx.x;
    const uint32_t least = t.link_bits > t.hs ? 1u << (t.link_bits - t.hs) : 1u;
    const uint32_t N = min(max(next_pow2(r_len), max(least, 4u)), t.hcap);
    t.mask = N - 1;
    t.tag_shift = t.hs + 31 - __clz(N);
    for (uint32_t i = tid; i < N / 4; i += THREADS)
        reinterpret_cast<uint4 *>(t.heads)[i] = make_uint4(CELL_EMPTY, CELL_EMPTY, CELL_EMPTY, CELL_EMPTY);
    __syncthreads();
    bool run = false;
    for (uint32_t i = tid; i < r_len; i += THREADS) {
        const uint32_t k = ld_key<CG>(R, r_off + i);
        uint32_t *head = &t.heads[(k >> t.hs) & t.mask];
        const uint32_t tag = t.tag_shift < 32 ? (k >> t.tag_shift) << t.link_bits : 0u;
        uint32_t old = *head;
        if (atomicCAS(head, old, old == CELL_EMPTY ? tag : tag | (i + 1)) != old) old = atomicExch(head, tag | (i + 1));
        if (old != CELL_EMPTY) {
            t.cells[i] = old;
            if (RUNS) run |= (old ^ tag) >> t.link_bits == 0;
        }
    }
    if (RUNS == RUNS_NONE) {
        __syncthreads();
    } else if (__syncthreads_or(run)) {
        auto look = RUNS == RUNS_CALL ? collapse_runs_call<THREADS, CG, E> : collapse_runs<THREADS, CG, E>;
        t.has_runs = look(t.heads, t.cells, t.mask, t.hs, t.link_bits, R + r_off, r_len, t.runs);
    } else {
        t.has_runs = false;
    }
}

// E: rows, or bare keys (layout 1 without payloads).
template <int THREADS, bool CG = false, class E = Row>
__device__ void build_table(Table &t, const E *__restrict__ R, uint64_t r_off, uint32_t r_len,
                            uint64_t *scan_scratch) {
    const int tid = threadIdx.x;
    constexpr bool ROWS = sizeof(E) == sizeof(Row);
    if (ROWS && t.layout == 0) {
        // next_pow2(|R_p|) buckets as in the reference, at most hcap (a
        // longer average chain when capR is not a power of two)
        const uint32_t N = min(next_pow2(r_len), t.hcap);
        t.mask = N - 1;
        for (uint32_t i = tid; i < r_len; i += THREADS) {
            const uint2 x = ld_elem<CG>(R, r_off + i);
            t.key[i] = x.x;
            t.pay[i] = x.y;
        }
        for (uint32_t i = tid; i < N; i += THREADS) t.heads[i] = 0;
        __syncthreads();
        for (uint32_t i = tid; i < r_len; i += THREADS) {
            uint32_t b = t.bucket(t.key[i]);
            t.next[i] = (uint16_t)atomicExch(&t.heads[b], i + 1);
        }
        __syncthreads();
    } else {
        uint32_t Nb = next_pow2(r_len) >> 2;
        if (Nb < 4) Nb = 4;
        t.mask = Nb - 1;
        uint32_t *cnt = t.heads;            // [Nb + 1]
        uint32_t *cur = t.heads + Nb + 1;   // cursors, Nb entries (fits: capR + 2 >= 2 Nb + 1)
        for (uint32_t i = tid; i <= Nb; i += THREADS) cnt[i] = 0;
        __syncthreads();
        for (uint32_t i = tid; i < r_len; i += THREADS)
            atomicAdd(&cnt[t.bucket(ld_elem<CG>(R, r_off + i).x)], 1u);
        __syncthreads();
        // exclusive scan of cnt[0..Nb) in place, cnt[Nb] = r_len
        const uint32_t per = (Nb + THREADS - 1) / THREADS;
        const uint32_t lo = min(Nb, tid * per), hi = min(Nb, lo + per);
        uint64_t s = 0;
        for (uint32_t i = lo; i < hi; i++) s += cnt[i];
        uint64_t tot;
        uint64_t run = block_excl_scan<THREADS>(s, &tot, scan_scratch);
        for (uint32_t i = lo; i < hi; i++) {
            uint32_t c = cnt[i];
            cnt[i] = (uint32_t)run;
            cur[i] = (uint32_t)run;
            run += c;
        }
        if (tid == 0) cnt[Nb] = r_len;
        __syncthreads();
        for (uint32_t i = tid; i < r_len; i += THREADS) {
            const uint2 x = ld_elem<CG>(R, r_off + i);
            uint32_t pos = atomicAdd(&cur[t.bucket(x.x)], 1u);
            t.key[pos] = x.x;
            if (ROWS && t.pay) t.pay[pos] = x.y;  // counting tables keep keys only
        }
        __syncthreads();
    }
}

// Sum of fn(key) over rows [0, len) (row pointer s, any 8-byte alignment),
// this thread's share: 16-byte loads, four in flight, and with
// TBG_PROBE_AHEAD the next group of four issued before the current group is
// looked up (the loads of one group then overlap the lookups of the previous).
#ifndef TBG_PROBE_AHEAD
#define TBG_PROBE_AHEAD 1
#endif
template <int THREADS, bool CG = false, class Fn>
__device__ __forceinline__ unsigned long long stream_sum(const Row *s, uint64_t len, Fn fn) {
    unsigned long long local = 0;
    const uint64_t head = ((reinterpret_cast<uintptr_t>(s) & 15) && len) ? 1 : 0;
    const uint64_t body = len - head;
    const uint64_t nv = body / 2;
    const bool tail = body & 1;
    const uint4 *v = reinterpret_cast<const uint4 *>(s + head);
    const int tid = threadIdx.x;
    if (head && tid == 0) local += fn(ld_row<CG>(s, 0).x);
    if (tail && tid == THREADS - 1) local += fn(ld_row<CG>(s, len - 1).x);
    uint64_t i = tid;
    if (TBG_PROBE_AHEAD && i + 3 * THREADS < nv) {
        uint4 n0 = ld_pair<CG>(v + i), n1 = ld_pair<CG>(v + i + THREADS);
        uint4 n2 = ld_pair<CG>(v + i + 2 * THREADS), n3 = ld_pair<CG>(v + i + 3 * THREADS);
        for (;;) {
            const uint4 x0 = n0, x1 = n1, x2 = n2, x3 = n3;
            i += 4 * THREADS;
            const bool more = i + 3 * THREADS < nv;
            if (more) {
                n0 = ld_pair<CG>(v + i);
                n1 = ld_pair<CG>(v + i + THREADS);
                n2 = ld_pair<CG>(v + i + 2 * THREADS);
                n3 = ld_pair<CG>(v + i + 3 * THREADS);
            }
            local += fn(x0.x) + fn(x0.z) + fn(x1.x) + fn(x1.z);
            local += fn(x2.x) + fn(x2.z) + fn(x3.x) + fn(x3.z);
            if (!more) break;
        }
    }
    for (; i + 3 * THREADS < nv; i += 4 * THREADS) {
        uint4 x0 = ld_pair<CG>(v + i), x1 = ld_pair<CG>(v + i + THREADS);
        uint4 x2 = ld_pair<CG>(v + i + 2 * THREADS), x3 = ld_pair<CG>(v + i + 3 * THREADS);
        local += fn(x0.x) + fn(x0.z) + fn(x1.x) + fn(x1.z);
        local += fn(x2.x) + fn(x2.z) + fn(x3.x) + fn(x3.z);
    }
    for (; i < nv; i += THREADS) {
        uint4 x0 = ld_pair<CG>(v + i);
        local += fn(x0.x) + fn(x0.z);
    }
    return local;
}

// Sum of fn(key) over the bare keys [0, len) of s (any alignment), this
// thread's share: 16-byte loads, two in flight while two are looked up.
template <int THREADS, bool CG = false, class Fn>
__device__ __forceinline__ unsigned long long stream_sum(const uint32_t *s, uint64_t len, Fn fn) {
    unsigned long long local = 0;
    const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(s) & 15) / 4;
    const uint32_t head = mis ? (uint32_t)umin64(4 - mis, len) : 0u;
    const uint64_t nv = (len - head) / 4;
    const uint32_t tail = (uint32_t)(len - head) & 3;
    const uint4 *v = reinterpret_cast<const uint4 *>(s + head);
    const uint32_t tid = threadIdx.x;
    if (tid < head) local += fn(ld_key<CG>(s, tid));
    if (tid < tail) local += fn(ld_key<CG>(s, len - 1 - tid));
    auto four = [&](const uint4 &x) { local += fn(x.x) + fn(x.y) + fn(x.z) + fn(x.w); };
    uint64_t i = tid;
    if (i + THREADS < nv) {
        uint4 n0 = ld_pair<CG>(v + i), n1 = ld_pair<CG>(v + i + THREADS);
        for (;;) {
            const uint4 x0 = n0, x1 = n1;
            i += 2 * THREADS;
            const bool more = i + THREADS < nv;
            if (more) {
                n0 = ld_pair<CG>(v + i);
                n1 = ld_pair<CG>(v + i + THREADS);
            }
            four(x0);
            four(x1);
            if (!more) break;
        }
    }
    for (; i < nv; i += THREADS) four(ld_pair<CG>(v + i));
    return local;
}

// Matches of S rows [0, len) against the table, this thread's share.
template <int THREADS, bool CG = false, class T = Table, class E = Row>
__device__ __forceinline__ unsigned long long probe_count(const T &t, const E *s, uint64_t len) {
    return stream_sum<THREADS, CG>(s, len, [&](uint32_t k) { return t.count(k); });
}

}  // namespace tbg
