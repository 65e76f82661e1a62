// Batched joins in one persistent launch.
//
// Every CTA pulls tickets from one counter; the ticket ranges are, in order,
//   build    one part of one join's bit table (direct joins, below);
//   probe    one chunk of the S_i of a join with a bit table;
//   hist     one chunk (`chunk` rows) of R_i or S_i: shared-memory histogram
//            over the join's P = 2^B partitions (low key bits);
//   scan     one join: column prefix of its chunk histograms (in place),
//            partition bases, join work items (S_p split every capS rows);
//   scatter  one chunk: the TMA-fed digit-sorting tile scatter of the
//            single-join partitioner, cursors = base[f] + prefix[chunk][f];
//   join     one worker of a partitioned join (pulls that join's items) or
//            one S slice of an unpartitioned join (B = 0, R_i loaded whole);
// build/probe runs out of shared memory as in the single-join kernel.  A
// ticket waits only on tickets handed out before it (per-join counters with
// acquire/release), so there is no grid-wide barrier and no co-residency
// requirement.  Data written earlier in the launch (histograms, bases,
// items, partitioned rows) is read with L2-only loads.
//
// Direct joins: when R_i's keys are distinct and lie in a compact range, one
// bit per key value is its whole hash table (direct.cu).  A build ticket
// enters R_i's keys into shared memory, where a key that is already there
// shows a duplicate, and writes the bits out; a probe ticket looks rows of S_i
// up in a copy of the bits.  S_i is read once and nothing is written.  The
// other tickets pass over the joins that are direct, and a CTA ends at the
// first of them when all are.  Bound by reading R and S: 512 joins of 2^10 ..
// 2^18 R rows, 228 M rows in all, take 0.46 ms (4.0 TB/s) against 1.89 ms
// partitioned.
//
// Each join's count equals the reference's RHO count on that join
// (Joins/radix_join.c:1558-1561, join_init_run :1237-1396; bucket
// chaining :187-244, histogram join :374-440).
#include <algorithm>

#include "batch.h"
#include "join_dev.cuh"
#include "part_dev.cuh"

namespace tbg {

namespace {

using BPart = PartSmem<BATCH_THREADS>;
static_assert(((size_t)1 << (BATCH_PART_LOG2 - 3)) <= sizeof(BPart), "a part of a bit table fits");

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Thread 0 waits until *flag >= target (bounded: records TBG_ERR_TIMEOUT and
// gives up), then the whole CTA proceeds.
__device__ void cta_wait(const unsigned *flag, unsigned target, unsigned *err) {
    if (threadIdx.x == 0) {
        unsigned ns = 32;
        for (uint32_t it = 0; ld_acquire_u32(flag) < target; it++) {
            if (it >= BATCH_SPIN_LIMIT) {
                atomicCAS(err, 0u, (unsigned)TBG_ERR_TIMEOUT);
                break;
            }
            __nanosleep(ns);
            if (ns < 512) ns <<= 1;
        }
        __threadfence();
    }
    __syncthreads();
}

// Publishes every write of this CTA, then *flag += 1.
__device__ void cta_signal(unsigned *flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(flag, 1u);
    }
}

__device__ __forceinline__ int ilog2(uint32_t p) { return 31 - __clz(p); }

// ---------------------------------------------------------------------------
// direct joins
// ---------------------------------------------------------------------------

// fn(key) for the rows [0, n) of s, this thread's share, 8 rows in flight (a
// plain loop: the other tickets' code leaves few registers free).
template <class Fn>
__device__ __forceinline__ void stream_keys(const Row *s, uint32_t n, Fn fn) {
    constexpr uint32_t T = BATCH_THREADS;
    const uint32_t head = (reinterpret_cast<uintptr_t>(s) & 15) && n ? 1u : 0u;
    const uint32_t nv = (n - head) / 2;
    const uint4 *v = reinterpret_cast<const uint4 *>(s + head);
    if (threadIdx.x == 0) {
        if (head) fn(s[0].key);
        if ((n - head) & 1) fn(s[n - 1].key);
    }
    uint32_t i = threadIdx.x;
    for (; i + 3 * T < nv; i += 4 * T) {
        const uint4 a = ldg_stream(v + i), b = ldg_stream(v + i + T), c = ldg_stream(v + i + 2 * T),
                    d = ldg_stream(v + i + 3 * T);
        fn(a.x), fn(a.z), fn(b.x), fn(b.z), fn(c.x), fn(c.z), fn(d.x), fn(d.z);
    }
    for (; i < nv; i += T) {
        const uint4 a = ldg_stream(v + i);
        fn(a.x), fn(a.z);
    }
}

__device__ __forceinline__ void block_min_max(uint32_t lo, uint32_t hi, uint32_t *red) {
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&red[0], lo);
        atomicMax(&red[1], hi);
    }
    __syncthreads();
}

// Part `bt.y` of a join's bit table: the bits [bt.y * 2^BATCH_PART_LOG2, ...) of it.
// A sample of R (the same for every part) that is wider than the table ends
// the attempt before R is read.  The last part to finish decides.
__device__ void build_part(const BatchArgs &a, uint32_t q, uint32_t *bits, uint32_t *red) {
    const uint2 bt = a.builds[q];
    const BatchJoin &J = a.joins[bt.x];
    BatchSync &sy = a.sync[bt.x];
    const int tid = threadIdx.x;
    const uint32_t w = J.bits_log2, mask = (1u << w) - 1;
    const uint32_t part_log2 = min(w, (uint32_t)BATCH_PART_LOG2), words = 1u << (part_log2 - 5);
    if (tid == 0) {
        red[0] = ~0u;
        red[1] = 0;
    }
    __syncthreads();
    {
        const uint64_t n = J.nR;
        const uint64_t i = n <= BATCH_THREADS ? tid : (uint64_t)tid * (n - 1) / (BATCH_THREADS - 1);
        const uint32_t k = i < n ? J.R[i].key : J.R[0].key;
        block_min_max(k, k, red);
    }
    if (red[1] - red[0] > mask) {
        if (tid == 0) atomicExch(&sy.off, 1u);
    } else {
        for (uint32_t i = tid; i < words; i += BATCH_THREADS) bits[i] = 0;
        __syncthreads();
        uint32_t lo = ~0u, hi = 0;
        bool dup = false;
        stream_keys(J.R, (uint32_t)J.nR, [&](uint32_t k) {
            lo = min(lo, k);
            hi = max(hi, k);
            const uint32_t s = k & mask;
            if (s >> part_log2 == bt.y) {
                const uint32_t b = s & ((1u << part_log2) - 1), bit = 1u << (b & 31);
                dup |= (atomicOr(&bits[b >> 5], bit) & bit) != 0;
            }
        });
        if (dup) atomicExch(&sy.off, 1u);
        __syncthreads();
        block_min_max(lo, hi, red);  // the sample's range lies inside R's
        if (tid == 0) {
            atomicMax(&sy.inv_min, ~red[0]);
            atomicMax(&sy.kmax, red[1]);
        }
        uint4 *dst = reinterpret_cast<uint4 *>(J.bits + (size_t)bt.y * words);
        for (uint32_t i = tid; i < words / 4; i += BATCH_THREADS) __stcg(dst + i, reinterpret_cast<uint4 *>(bits)[i]);
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        const uint32_t parts = 1u << (w - part_log2);
        if (atomicAdd(&sy.build_done, 1u) == parts - 1) {
            __threadfence();
            const bool ok = !__ldcg(&sy.off) && __ldcg(&sy.kmax) - ~__ldcg(&sy.inv_min) <= mask;
            if (ok) atomicAdd(a.direct, 1u);
            __threadfence();
            atomicExch(&sy.decision, ok ? 1u : 2u);
        }
    }
}

// Whether join j is direct (the same for every thread); waits for its bit
// table's decision.
template <bool DIRECT>
__device__ __forceinline__ bool is_direct(const BatchArgs &a, uint32_t j) {
    if (!DIRECT || !a.joins[j].bits) return false;
    cta_wait(&a.sync[j].decision, 1, a.err);
    return __ldcg(&a.sync[j].decision) == 1;
}

// Matches of one chunk of a direct join's S: bits from a copy in shared
// memory (`cap` words), or from L2 when R's range is wider.
__device__ void direct_chunk(const BatchArgs &a, uint32_t q, uint32_t *copy, uint32_t cap) {
    const uint2 c = a.dchunks[q];
    const uint32_t j = c.x;
    if (!is_direct<true>(a, j)) return;
    const BatchJoin &J = a.joins[j];
    const uint64_t lo = (uint64_t)c.y * BATCH_DCHUNK, hi = umin64(J.nS, lo + BATCH_DCHUNK);
    const uint32_t kmin = ~__ldcg(&a.sync[j].inv_min), span = __ldcg(&a.sync[j].kmax) - kmin;
    const uint32_t wordmask = (1u << (J.bits_log2 - 5)) - 1, w0 = kmin >> 5;
    const uint32_t words = ((kmin + span) >> 5) - w0 + 1;
    const uint32_t *bits = J.bits;
    uint32_t local = 0;  // a chunk holds BATCH_DCHUNK rows at most
    if (words <= cap) {
        for (uint32_t i = threadIdx.x; i < words; i += BATCH_THREADS) copy[i] = __ldcg(bits + ((w0 + i) & wordmask));
        __syncthreads();
        stream_keys(J.S + lo, (uint32_t)(hi - lo), [&](uint32_t k) {
            if (k - kmin <= span) local += (copy[(k >> 5) - w0] >> (k & 31)) & 1u;
        });
    } else {
        stream_keys(J.S + lo, (uint32_t)(hi - lo), [&](uint32_t k) {
            if (k - kmin <= span) local += (__ldcg(bits + ((k >> 5) & wordmask)) >> (k & 31)) & 1u;
        });
    }
    local = __reduce_add_sync(0xffffffffu, local);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(a.counts + J.orig, (unsigned long long)local);
}

// ---------------------------------------------------------------------------
// hist: chunk histogram over the join's partitions
// ---------------------------------------------------------------------------
// Per-warp sub-histograms (P <= 256 bins each): with so few bins nearly every
// warp holds repeated digits, so each row pays one shared atomic on its
// warp's own bins instead of a match-based aggregation; the warps' bins are
// summed at the end of the chunk.
__device__ void hist_chunk(const BatchArgs &a, uint32_t c, uint32_t *bins) {
    constexpr int NW = BATCH_THREADS / 32;
    const uint2 ch = a.chunks[c];
    const BatchJoin &J = a.joins[ch.x];
    const int rel = ch.y >> 31;
    const uint32_t idx = ch.y & 0x7fffffffu;
    const Row *in = rel ? J.S : J.R;
    const uint64_t n = rel ? J.nS : J.nR;
    const uint32_t P = J.P, mask = P - 1;
    const int tid = threadIdx.x;
    uint32_t *wb = bins + (tid >> 5) * BATCH_FMAX;  // this warp's bins
    for (uint32_t i = tid; i < NW * BATCH_FMAX; i += BATCH_THREADS) bins[i] = 0;
    __syncthreads();
    const uint64_t lo = (uint64_t)idx * J.chunk;
    const uint64_t hi = umin64(n, lo + J.chunk);
    const uint64_t head = ((reinterpret_cast<uintptr_t>(in + lo) & 15) != 0) ? 1 : 0;
    const uint64_t body = hi - lo - head;
    const uint64_t nv = body / 2;
    const uint4 *v = reinterpret_cast<const uint4 *>(in + lo + head);
    const uint64_t per = (uint64_t)BATCH_THREADS * 4;
    for (uint64_t base = 0; base < nv; base += per) {
        uint4 x[4];
        bool ok[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint64_t i = base + (uint64_t)u * BATCH_THREADS + tid;
            ok[u] = i < nv;
            if (ok[u]) x[u] = ldg_stream(v + i);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (ok[u]) {
                atomicAdd(&wb[x[u].x & mask], 1u);
                atomicAdd(&wb[x[u].z & mask], 1u);
            }
        }
    }
    if (tid == 0) {
        if (head) atomicAdd(&wb[in[lo].key & mask], 1u);
        if (body & 1) atomicAdd(&wb[in[hi - 1].key & mask], 1u);
    }
    __syncthreads();
    uint32_t *dst = (rel ? J.histS : J.histR) + (uint64_t)idx * P;
    for (uint32_t f = tid; f < P; f += BATCH_THREADS) {
        uint32_t t = 0;
#pragma unroll
        for (int w = 0; w < NW; w++) t += bins[w * BATCH_FMAX + f];
        __stcg(dst + f, t);
    }
    cta_signal(&a.sync[ch.x].hist_done);
}

// ---------------------------------------------------------------------------
// scan: column prefix, bases, items
// ---------------------------------------------------------------------------

// In place: h[c][f] <- sum_{c' < c} h[c'][f]; tot[f] <- column total.
// Thread (z, f) owns chunk segment z of column f.
__device__ void column_prefix(uint32_t *h, uint32_t G, uint32_t P, uint32_t *part, uint32_t *tot) {
    const int tid = threadIdx.x;
    const int lp = ilog2(P);
    const uint32_t Z = BATCH_THREADS >> lp;
    const uint32_t f = tid & (P - 1), z = tid >> lp;
    const uint32_t seg = (G + Z - 1) / Z;
    const uint32_t c0 = min(G, z * seg), c1 = min(G, c0 + seg);
    uint32_t s = 0;
    uint32_t c = c0;
    for (; c + 8 <= c1; c += 8) {
        uint32_t x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = __ldcg(h + (uint64_t)(c + u) * P + f);
#pragma unroll
        for (int u = 0; u < 8; u++) s += x[u];
    }
    for (; c < c1; c++) s += __ldcg(h + (uint64_t)c * P + f);
    part[tid] = s;
    __syncthreads();
    uint32_t run = 0;
    for (uint32_t zz = 0; zz < z; zz++) run += part[zz * P + f];
    if (z == 0) {
        uint32_t t = 0;
        for (uint32_t zz = 0; zz < Z; zz++) t += part[zz * P + f];
        tot[f] = t;
    }
    c = c0;
    for (; c + 8 <= c1; c += 8) {
        uint32_t x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = __ldcg(h + (uint64_t)(c + u) * P + f);
#pragma unroll
        for (int u = 0; u < 8; u++) {
            __stcg(h + (uint64_t)(c + u) * P + f, run);
            run += x[u];
        }
    }
    for (; c < c1; c++) {
        const uint32_t x = __ldcg(h + (uint64_t)c * P + f);
        __stcg(h + (uint64_t)c * P + f, run);
        run += x;
    }
    __syncthreads();
}

__device__ void scan_join(const BatchArgs &a, uint32_t q, uint32_t *sm, uint64_t *scratch) {
    const uint32_t j = a.scans[q];
    const BatchJoin &J = a.joins[j];
    cta_wait(&a.sync[j].hist_done, J.GR + J.GS, a.err);
    const int tid = threadIdx.x;
    const uint32_t P = J.P;
    uint32_t *part = sm;                          // [BATCH_THREADS]
    uint32_t *tot = part + BATCH_THREADS;         // [2][BATCH_FMAX]
    uint32_t *base = tot + 2 * BATCH_FMAX;        // [2][BATCH_FMAX]
    column_prefix(J.histR, J.GR, P, part, tot);
    column_prefix(J.histS, J.GS, P, part, tot + BATCH_FMAX);
    bool ok = true;
    for (int rel = 0; rel < 2; rel++) {
        uint64_t total;
        const uint32_t x = (uint32_t)tid < P ? tot[rel * BATCH_FMAX + tid] : 0;
        const uint64_t b = block_excl_scan<BATCH_THREADS>(x, &total, scratch);
        if ((uint32_t)tid < P) {
            base[rel * BATCH_FMAX + tid] = (uint32_t)b;
            __stcg((rel ? J.baseS : J.baseR) + tid, (uint32_t)b);
        }
        // every chunk histogram landed exactly once: totals add up to |rel|
        ok = ok && total == (rel ? J.nS : J.nR);
    }
    __syncthreads();
    uint32_t rl = 0, sl = 0, ns = 0;
    if ((uint32_t)tid < P) {
        rl = tot[tid];
        sl = tot[BATCH_FMAX + tid];
        ns = (rl && sl) ? (sl + J.capS - 1) / J.capS : 0;
    }
    uint64_t nit;
    const uint64_t pos = block_excl_scan<BATCH_THREADS>(ns, &nit, scratch);
    if (!ok || nit > J.item_cap) {
        // only reachable after a wait above gave up
        if (tid == 0) atomicCAS(a.err, 0u, (unsigned)TBG_ERR_TIMEOUT);
        nit = 0;
    } else {
        for (uint32_t k = 0; k < ns; k++) {
            Item m;
            m.r_off = base[tid];
            m.r_len = rl;
            m.s_off = (uint64_t)base[BATCH_FMAX + tid] + (uint64_t)k * J.capS;
            m.s_len = min(J.capS, sl - k * J.capS);
            m.part = tid;
            J.items[pos + k] = m;
        }
    }
    if (tid == 0) __stcg(&a.sync[j].nitems, (unsigned)nit);
    cta_signal(&a.sync[j].scan_done);
}

// ---------------------------------------------------------------------------
// scatter: one chunk into its join's partitions
// ---------------------------------------------------------------------------
__device__ void scatter_chunk(const BatchArgs &a, uint32_t c, BPart &sm, uint64_t *mbar, uint32_t &kseq) {
    const uint2 ch = a.chunks[c];
    const BatchJoin &J = a.joins[ch.x];
    cta_wait(&a.sync[ch.x].scan_done, 1, a.err);
    const int rel = ch.y >> 31;
    const uint32_t idx = ch.y & 0x7fffffffu;
    const uint32_t P = J.P;
    const uint32_t *base = rel ? J.baseS : J.baseR;
    const uint32_t *pre = (rel ? J.histS : J.histR) + (uint64_t)idx * P;
    for (uint32_t f = threadIdx.x; f < P; f += BATCH_THREADS) sm.cursor[f] = __ldcg(base + f) + __ldcg(pre + f);
    const Row *in = rel ? J.S : J.R;
    const uint64_t n = rel ? J.nS : J.nR;
    const uint64_t lo = (uint64_t)idx * J.chunk;
    const uint64_t hi = umin64(n, lo + J.chunk);
    part_tiles<BATCH_THREADS, uint32_t>(in, lo, hi, n, rel ? J.Sp : J.Rp, (uint32_t)n, DigitOp{0u, P - 1}, sm, mbar,
                                        kseq, a.err);
    cta_signal(&a.sync[ch.x].scat_done);
}

// ---------------------------------------------------------------------------
// join: build/probe
// ---------------------------------------------------------------------------
// R and S: the caller's rows, or (CG, written earlier in the launch)
// partitions of bare keys.
template <bool CG, class E>
__device__ unsigned long long pair_count(Table &t, CellTable &ct, const E *R, uint64_t rn, const E *S, uint64_t sn,
                                         uint32_t capR, uint64_t *scratch) {
    unsigned long long c = 0;
    for (uint64_t r0 = 0; r0 < rn; r0 += capR) {
        const uint32_t n = (uint32_t)umin64(capR, rn - r0);
        if (t.layout == 0) {
            build_cells<BATCH_THREADS, CG>(ct, R, r0, n);
            c += probe_count<BATCH_THREADS, CG>(ct, S, sn);
        } else {
            build_table<BATCH_THREADS, CG>(t, R, r0, n, scratch);
            c += probe_count<BATCH_THREADS, CG>(t, S, sn);
        }
        __syncthreads();  // table rebuilt by the next R slice
    }
    return c;
}

__device__ void join_ticket(const BatchArgs &a, uint32_t q, unsigned char *smem, uint64_t *scratch,
                            uint32_t *s_item) {
    const uint2 jt = a.jt[q];
    const BatchJoin &J = a.joins[jt.x];
    const uint32_t capR = a.capR;
    Table t;  // layout 1 (histogram table)
    t.key = reinterpret_cast<uint32_t *>(smem);
    t.pay = t.key + capR;
    t.heads = t.pay + capR;
    t.next = nullptr;
    t.hs = (int)J.B;
    t.layout = (int)J.layout;
    t.hcap = floor_pow2(capR + 2);
    CellTable ct;  // layout 0 (bucket chains)
    ct.link_bits = cell_link_bits(capR);
    ct.hcap = 1u << ct.link_bits;  // an unpartitioned join (B = 0) needs them all
    ct.heads = reinterpret_cast<uint32_t *>(smem);
    ct.cells = ct.heads + ct.hcap;
    ct.hs = (int)J.B;
    unsigned long long local = 0;
    if (J.B == 0) {
        const uint64_t lo = (uint64_t)jt.y * J.capS;
        const uint64_t hi = umin64(J.nS, lo + J.capS);
        if (lo < hi) local = pair_count<false>(t, ct, J.R, J.nR, J.S + lo, hi - lo, capR, scratch);
    } else {
        BatchSync &sy = a.sync[jt.x];
        cta_wait(&sy.scat_done, J.GR + J.GS, a.err);
        const unsigned nit = __ldcg(&sy.nitems);
        for (;;) {
            if (threadIdx.x == 0) *s_item = atomicAdd(&sy.item_ctr, 1u);
            __syncthreads();
            const unsigned i = *s_item;
            __syncthreads();
            if (i >= nit) break;
            const uint4 *mp = reinterpret_cast<const uint4 *>(J.items + i);
            const uint4 m0 = __ldcg(mp), m1 = __ldcg(mp + 1);
            const uint64_t r_off = (uint64_t)m0.x | ((uint64_t)m0.y << 32);
            const uint64_t s_off = (uint64_t)m0.z | ((uint64_t)m0.w << 32);
            const uint64_t s_len = (uint64_t)m1.x | ((uint64_t)m1.y << 32);
            const uint32_t r_len = m1.z;
            if (r_off + r_len <= J.nR && s_off + s_len <= J.nS)
                local += pair_count<true>(t, ct, J.Rp + r_off, r_len, J.Sp + s_off, s_len, capR, scratch);
        }
    }
    const unsigned long long ws = warp_sum_u64(local);
    if ((threadIdx.x & 31) == 0 && ws) atomicAdd(a.counts + J.orig, ws);
}

static_assert(sizeof(Item) == 32, "join_ticket reads an item as two 16-byte words");

}  // namespace

// DIRECT: the plan has bit tables.
template <bool DIRECT>
__global__ void __launch_bounds__(BATCH_THREADS, 2) k_batch(BatchArgs a, uint32_t smem_words) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t mbar[PART_NBUF];
    __shared__ uint64_t scratch[BATCH_THREADS / 32 + 1];
    __shared__ uint32_t s_ticket, s_item, s_red[2];
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int i = 0; i < PART_NBUF; i++) mbar_init(&mbar[i], 1);
        fence_mbar_init();
    }
    uint32_t kseq = 0;
    const uint32_t t_hist = DIRECT ? a.n_builds + a.n_dchunks : 0u, t_scan = t_hist + a.n_chunks;
    const uint32_t t_scat = t_scan + a.n_scans, t_join = t_scat + a.n_chunks, t_end = t_join + a.n_jt;
    for (;;) {
        if (tid == 0) {
            uint32_t t = atomicAdd(a.ticket, 1u);
            if (DIRECT && t >= t_hist && ld_acquire_u32(a.direct) == a.njoins) t = t_end;  // nothing is left to do
            s_ticket = t;
        }
        __syncthreads();
        const uint32_t t = s_ticket;
        __syncthreads();
        if (t >= t_end) break;
        if (DIRECT && t < t_hist) {
            if (t < a.n_builds) build_part(a, t, reinterpret_cast<uint32_t *>(smem), s_red);
            else direct_chunk(a, t - a.n_builds, reinterpret_cast<uint32_t *>(smem), smem_words);
        } else {
            // the join of this ticket
            const uint32_t j = t < t_scan ? a.chunks[t - t_hist].x
                             : t < t_scat ? a.scans[t - t_scan]
                             : t < t_join ? a.chunks[t - t_scat].x
                                          : a.jt[t - t_join].x;
            if (is_direct<DIRECT>(a, j)) continue;
            if (t < t_scan) hist_chunk(a, t - t_hist, reinterpret_cast<uint32_t *>(smem));
            else if (t < t_scat) scan_join(a, t - t_scan, reinterpret_cast<uint32_t *>(smem), scratch);
            else if (t < t_join) scatter_chunk(a, t - t_scat, *reinterpret_cast<BPart *>(smem), mbar, kseq);
            else join_ticket(a, t - t_join, smem, scratch, &s_item);
        }
        __syncthreads();  // shared memory is reused by the next ticket
    }
}

size_t batch_smem_bytes() {
    size_t s = sizeof(BPart);
    const size_t j = join_smem_bytes(BATCH_CAPR);
    if (j > s) s = j;
    const size_t sc = std::max<size_t>(BATCH_THREADS + 4 * BATCH_FMAX, BATCH_THREADS / 32 * BATCH_FMAX) * sizeof(uint32_t);
    if (sc > s) s = sc;
    return s;
}

cudaError_t batch_occupancy(int *per_sm) {
    const size_t smem = batch_smem_bytes();
    int n = 0;
    cudaError_t e = smem_limit((const void *)k_batch<false>, smem);
    if (e == cudaSuccess) e = smem_limit((const void *)k_batch<true>, smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_batch<true>, BATCH_THREADS, smem);
    if (e != cudaSuccess) return e;
    *per_sm = n < 1 ? 1 : n;
    return cudaSuccess;
}

int batch_ctas_per_sm() {
    int n = 1;
    if (batch_occupancy(&n) != cudaSuccess) cudaGetLastError();
    return n;
}

// batch_ctas_per_sm() (called when a plan is made, outside any stream
// capture) sets the kernel's shared-memory attribute.
cudaError_t launch_batch(const BatchArgs &a, int grid, cudaStream_t st) {
    const size_t smem = batch_smem_bytes();
    auto kern = a.n_builds ? k_batch<true> : k_batch<false>;
    kern<<<grid, BATCH_THREADS, smem, st>>>(a, (uint32_t)(smem / 4));
    count_launch();
    return cudaGetLastError();
}

}  // namespace tbg
