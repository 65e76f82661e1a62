// Joins with a small R in one launch.
//
// With at most SMALL_R rows R's whole table fits one CTA's shared memory, so
// every CTA builds it from R (read from L2) and joins its slice of S with it:
// nothing is histogrammed, planned or partitioned, and no launch follows
// another.  The partitioned join of 3000 x 20011 rows is eleven launches of 2
// to 11 us each (83 us in all from Python); this is one.
//
// Counting, the table is one bit per key value when R's keys are distinct and
// their range fits shared memory (as in direct.cu), else the bucket chains of
// the partitioned join (join_dev.cuh; Joins/radix_join.c:187-244), long runs of
// one key counted: 4000 rows of one key x 1 M rows take 43 us, 4.7 ms along the
// chain (RSM's sorted merge, the other plan for it, 155 us).
// Materialising joins use bucket chains with payloads.  The last CTA to finish
// fills the control block, with the partition sizes and work items that the
// partitioned join would have had (a few partitions: 2 to 8), in device memory
// and in the caller's pinned mirror, so that no copy follows either.
#include <algorithm>
#include <type_traits>

#include "join_dev.cuh"
#include "tbg_runtime.h"

namespace tbg {

constexpr int SMALL_THREADS = 1024;
constexpr size_t SMALL_SMEM_MAX = 223 * 1024;

struct SmallArgs {
    const Row *R, *S;
    uint64_t nS, slice;       // S rows, rows per CTA
    uint32_t nR;
    int B;                    // radix bits of the statistics (P = 2^B <= 8)
    int capR;                 // rows of R per work item (statistics)
    SplitRule split;
    uint64_t item_cap;
    uint32_t table_rows;      // shared-memory table size
    uint32_t bit_words;       // words of shared memory for bits
    SmallCtl *sc;
    Ctrl *ctrl, *host;        // host: pinned mirror (null: the caller does not wait for it)
    tbg_row_out *out;
    uint64_t cap;
};

// Heads of the count-only table: two per row (2^13 at 4096 rows, 2^14, 2^15),
// as many as the tag needs.
__host__ __device__ __forceinline__ uint32_t small_heads(uint32_t table_rows) {
    return 1u << cell_link_bits(table_rows);
}

// Adds the block's counts of digits [0, P) of this thread's key to cnt[8]
// (shared); every lane of the warp calls it.
__device__ __forceinline__ void count_digits(uint32_t *cnt, uint32_t key, bool valid, int P) {
    for (int d = 0; d < P; d++) {
        const unsigned m = __ballot_sync(0xffffffffu, valid && (key & (P - 1)) == (uint32_t)d);
        if ((threadIdx.x & 31) == 0 && m) atomicAdd(&cnt[d], (uint32_t)__popc(m));
    }
}

template <bool MAT>
__global__ void __launch_bounds__(SMALL_THREADS, 1) k_small(SmallArgs a) {
    constexpr int T = SMALL_THREADS;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t scratch[T / 32 + 1];
    __shared__ uint32_t red[2], cnt[8], dup;
    __shared__ unsigned long long blk;
    __shared__ bool last;
    __shared__ Ctrl fin;
    const int tid = threadIdx.x, lane = tid & 31;
    const int P = 1 << a.B;
    if (tid < 8) cnt[tid] = 0;
    if (tid == 0) {
        red[0] = ~0u;
        red[1] = dup = 0;
        blk = 0;
    }
    __syncthreads();

    // R's table
    Table t;
    CellTable ct;
    __shared__ std::conditional_t<MAT, uint32_t, LongRuns> runs;
    if (MAT) {
        t.key = reinterpret_cast<uint32_t *>(smem);
        t.hs = 0;  // nothing is partitioned: keys differ in every bit
        t.layout = 0;
        t.pay = t.key + a.table_rows;
        t.heads = t.pay + a.table_rows;
        t.next = reinterpret_cast<uint16_t *>(t.heads + a.table_rows + 2);
        t.hcap = floor_pow2(a.table_rows + 2);
    } else {
        ct.hcap = small_heads(a.table_rows);
        ct.heads = reinterpret_cast<uint32_t *>(smem);
        ct.cells = ct.heads + ct.hcap;
        ct.hs = 0;
        ct.link_bits = cell_link_bits(a.table_rows);
        ct.runs = reinterpret_cast<LongRuns *>(&runs);
    }
    uint32_t *bits = reinterpret_cast<uint32_t *>(smem);
    uint32_t kmin = 0, span = 0;
    bool by_bits = false;
    if (!MAT) {
        uint32_t lo = ~0u, hi = 0;
        for (uint32_t i = tid; i < a.nR; i += T) {
            const uint32_t k = a.R[i].key;
            lo = min(lo, k);
            hi = max(hi, k);
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) {
            atomicMin(&red[0], lo);
            atomicMax(&red[1], hi);
        }
        __syncthreads();
        kmin = red[0];
        span = red[1] - kmin;
        if (span / 32 < a.bit_words && a.nR <= span + 1) {
            for (uint32_t i = tid; i <= span / 32; i += T) bits[i] = 0;
            __syncthreads();
            bool d = false;
            for (uint32_t i = tid; i < a.nR; i += T) {
                const uint32_t k = a.R[i].key - kmin, bit = 1u << (k & 31);
                d |= (atomicOr(&bits[k >> 5], bit) & bit) != 0;
            }
            if (d) dup = 1;
            __syncthreads();
            by_bits = dup == 0;
        }
    }
    if (MAT) build_table<T>(t, a.R, 0, a.nR, scratch);
    else if (!by_bits) build_cells<T, false, RUNS_INLINE>(ct, a.R, 0, a.nR);

    // this CTA's slice of S
    const uint64_t s0 = (uint64_t)blockIdx.x * a.slice;
    const uint64_t len = umin64(a.slice, a.nS - s0);
    const Row *s = a.S + s0;
    unsigned long long local = 0;
    if (!MAT) {
        uint32_t odd = 0;  // P = 2: the rows of partition 1 (a slice holds < 2^32 rows)
        if (by_bits) {
            local = stream_sum<T>(s, len, [&](uint32_t k) {
                odd += k & 1;
                const uint32_t d = k - kmin;
                return d <= span ? (bits[d >> 5] >> (d & 31)) & 1u : 0u;
            });
        } else if (!ct.has_runs) {
            local = stream_sum<T>(s, len, [&](uint32_t k) {
                odd += k & 1;
                return ct.count(k);
            });
        } else {
            local = stream_sum<T>(s, len, [&](uint32_t k) {
                odd += k & 1;
                return ct.count<true>(k);
            });
        }
        odd = __reduce_add_sync(0xffffffffu, odd);
        if (lane == 0 && odd) atomicAdd(&cnt[1], odd);
    } else {
        for (uint64_t b = 0; b < len; b += 4ull * T) {
            uint32_t k[4], p[4], c[4];
            uint64_t pos[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint64_t i = b + (uint64_t)u * T + tid;
                const bool ok = i < len;
                const uint2 x = ok ? ldg_stream(reinterpret_cast<const uint2 *>(s) + i) : make_uint2(0, 0);
                k[u] = x.x;
                p[u] = x.y;
                count_digits(cnt, x.x, ok, P);
                c[u] = ok ? t.count(x.x) : 0;
                local += c[u];
            }
            block_emit_positions<T, 4>(c, pos, &a.sc->rows, scratch);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (!c[u]) continue;
                uint64_t q = pos[u];
                t.for_each(k[u], [&](uint32_t rp) {
                    if (q < a.cap) a.out[q] = tbg_row_out{k[u], rp, p[u]};
                    q++;
                });
            }
        }
    }
    const unsigned long long ws = warp_sum_u64(local);
    if (lane == 0 && ws) atomicAdd(&blk, ws);
    __syncthreads();

    // the CTA's sums, then the last CTA's control block
    if (tid < P && cnt[tid]) atomicAdd(&a.sc->hist[tid], cnt[tid]);
    __syncthreads();
    if (tid == 0) {
        if (blk) atomicAdd(&a.sc->matches, blk);
        __threadfence();
        last = atomicAdd(&a.sc->done, 1u) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    if (tid < 8) cnt[tid] = 0;
    for (int i = tid; i < (int)(sizeof(Ctrl) / 4); i += T) reinterpret_cast<uint32_t *>(&fin)[i] = 0;
    __syncthreads();
    for (uint32_t i0 = 0; i0 < a.nR; i0 += T) {
        const bool ok = i0 + tid < a.nR;
        count_digits(cnt, ok ? a.R[i0 + tid].key : 0, ok, P);
    }
    __syncthreads();
    if (tid == 0) {
        uint32_t hs[8];
        uint64_t all = 0, items = 0;
        unsigned long long sum1 = 0;
        for (int f = 0; f < P; f++) {
            hs[f] = __ldcg(&a.sc->hist[f]);
            sum1 += hs[f];
        }
        if (!MAT) hs[0] = (uint32_t)(a.nS - sum1);  // counting adds up partition 1 only
        for (int pass = 0; pass < 2; pass++) {  // the planner's split decision, then its items (partition.cu)
            uint64_t n = 0;
            for (int f = 0; f < P; f++) {
                const uint32_t hr = cnt[f];
                if (!hr || !hs[f]) continue;
                const uint64_t nrc = (hr + (uint64_t)a.capR - 1) / a.capR;
                n += nrc * (pass && nrc > 1 && all > a.item_cap ? 1 : a.split.items(hs[f], nrc));
            }
            (pass ? items : all) = n;
        }
        for (int f = 0; f < P; f++) {
            fin.max_part_R = max(fin.max_part_R, (unsigned long long)cnt[f]);
            fin.max_part_S = max(fin.max_part_S, (unsigned long long)hs[f]);
            fin.nonempty += cnt[f] && hs[f];
        }
        fin.nitems = (unsigned)items;
        fin.matches = __ldcg(&a.sc->matches);
        fin.rows = __ldcg(&a.sc->rows);
    }
    __syncthreads();
    for (int i = tid; i < (int)(sizeof(Ctrl) / 4); i += T) {
        const uint32_t x = reinterpret_cast<uint32_t *>(&fin)[i];
        reinterpret_cast<uint32_t *>(a.ctrl)[i] = x;
        if (a.host) reinterpret_cast<uint32_t *>(a.host)[i] = x;
    }
    // the counters start the next launch at zero
    for (int i = tid; i < (int)(sizeof(SmallCtl) / 4); i += T) reinterpret_cast<uint32_t *>(a.sc)[i] = 0;
}

// Whether the join with radix geometry g is a small one.  Counting keeps the
// S rows of one of two partitions (any more would cost the probe loop).
bool is_small_join(const tbg_config &cfg, const RadixGeom &g) {
    return automatic_plan(cfg) && g.n[0] <= SMALL_R && (cfg.materialize ? g.P <= 8 : g.P == 2);
}

int run_small_join(const tbg_config &cfg, const RadixGeom &g, const Row *dR, const Row *dS, tbg_row_out *d_rows,
                   uint64_t cap, Workspace &w, cudaStream_t st, JoinRun *run) {
    const bool mat = cfg.materialize != 0;
    cudaError_t e = w.small.ensure(sizeof(SmallCtl));
    if (e == cudaSuccess && w.small.fresh) {
        e = cudaMemsetAsync(w.small.p, 0, sizeof(SmallCtl), st);
        w.small.fresh = e != cudaSuccess;
    }
    if (e != cudaSuccess) return cuda_error(e, "small join");
    const uint64_t nR = g.n[0], nS = g.n[1];
    SmallArgs a;
    a.R = dR;
    a.S = dS;
    a.nR = (uint32_t)nR;
    a.nS = nS;
    // one CTA per SM, at least 2048 rows each; a row may have to write all of R,
    // so rows that are written are spread over the SMs however few they are
    // (16000 R rows of 10 keys x 2000, 3.2 M rows out: 0.28 ms, 7.6 ms with
    // one CTA and a table that dropped the keys' low bits)
    a.slice = std::max<uint64_t>(mat ? 8 : 2048, (nS + w.nsm - 1) / w.nsm);
    a.B = g.B;
    a.capR = g.capR;
    a.split = g.split;
    a.item_cap = g.item_cap;
    a.table_rows = nR <= 4096 ? 4096 : nR <= 8192 ? 8192 : 16384;
    a.sc = w.small.as<SmallCtl>();
    a.ctrl = w.ctrl.as<Ctrl>();
    a.host = run->waits ? w.host_ctrl : nullptr;
    a.out = d_rows;
    a.cap = d_rows && mat ? cap : 0;
    const size_t smem = mat ? join_smem_bytes((int)a.table_rows)
                            : std::max(((size_t)small_heads(a.table_rows) + a.table_rows) * 4,
                                       std::min<size_t>(SMALL_SMEM_MAX, (size_t)nR * 4));  // 32 key values per row
    a.bit_words = mat ? 0 : (uint32_t)(smem / 4);
    auto kern = mat ? k_small<true> : k_small<false>;
    mark(w, cfg.timing != 0, 0, st);
    if ((e = smem_limit((const void *)kern, smem)) != cudaSuccess) return cuda_error(e, "small join");
    kern<<<(unsigned)((nS + a.slice - 1) / a.slice), SMALL_THREADS, smem, st>>>(a);
    count_launch();
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_error(e, "small join");
    for (int i = 1; i <= 4; i++) mark(w, cfg.timing != 0, i, st);
    run->timed = cfg.timing != 0;
    run->B = g.B;
    run->passes = g.passes;
    run->P = g.P;
    run->ctrl_on_host = run->waits;
    run->small = true;
    return TBG_OK;
}

}  // namespace tbg
