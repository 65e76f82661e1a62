// Direct counting join: when R's keys are distinct and lie in a compact
// range, one bit per key value is a perfect hash table of R that fits the L2
// cache (or shared memory), and S is joined while it is read for its
// histogram, without being partitioned.
//
// The reference's counting RHO and RHT (Joins/radix_join.c:187-244, :374-440)
// partition both relations so that every R partition's table fits a core's
// cache.  Here the bit table does: 2^27 keys are 16.8 MB, a seventh of the
// L2.  Counting needs no payloads, and a distinct key matches at most once,
// so the bit is the whole table entry.  For the sort-merge joins RSM and PSM
// the set bits are R's distinct keys in order, and S's rows are merged with
// them as they come.
//
// Bit of key k: k mod 2^w.  With max - min < 2^w that is injective on
// [min, max], so R can be entered while it is read for its histogram, before
// its range is known:
//   k_direct_prep   guesses w from a sample of R (no guess: not direct) and
//                   clears the table;
//   k_hist_build    R's chunk histograms (as k_hist_chunks), the key range,
//                   and the bits;
//   k_direct_decide counts the set bits: direct iff the range fits 2^w and
//                   |R| bits are set (all keys distinct);
//   k_hist_probe    S's chunk histograms, and with the decision the matches.
// A materialising join keeps R's payload per key value instead of a bit
// (k_hist_build<true>, k_hist_emit): 2^22 keys are 16.8 MB.  A payload equal to
// the empty mark, like a key that occurs twice, sends the join to the passes.
// The histograms are the partitioned join's own, so when the decision is no,
// the join continues with the passes, and the statistics (partition sizes,
// work items) are the same either way.
#include <algorithm>

#include "part_dev.cuh"
#include "tbg_runtime.h"

namespace tbg {

constexpr int DIRECT_THREADS = 1024;
constexpr int DIRECT_MIN_LOG2 = 10;
constexpr uint32_t EMPTY_PAYLOAD = 0xFFFFFFFFu;  // a key value that R does not hold

// log2 of the largest table considered for nR rows: 32 bits per row (a
// filtered or sparse key range up to 1/32 full), at most 2^29 bits (67 MB).
// Measured on 2^30 S rows: 4.02 ms for tables of 0.5 to 34 MB, 5.0 ms at
// 67 MB, 10.9 ms at 134 MB (out of the L2), where the partitioned join takes
// 11.4 ms or more.
int direct_log2_max(uint64_t nR) {
    int k = DIRECT_MIN_LOG2;
    while (k < 29 && (1ull << k) < nR * 32) k++;
    return k;
}

// Shared memory words for a CTA's copy of the bit table or of one of two parts
// of it: what a CTA can hold beside its histogram bins (one CTA per SM either
// way).  A table in shared memory is read at the speed of S's stream (2^30
// rows: 1.37 ms), one in L2 at one line per clock and SM (4.02 ms); in two
// parts every row is read twice, which is still faster than L2 (2.5 M x 50 M
// rows: 241 against 314 us), in three not (5 M x 100 M: 459 against 470 us,
// 5 M x 20 M: 175 against 168 us).  Zero when one bit per row would not fit.
constexpr uint32_t DIRECT_PARTS = 2;
uint32_t direct_smem_words(uint64_t nR, uint64_t nbins) {
    constexpr uint64_t CAP = 220 * 1024 / 4;
    if (nbins >= CAP / 2) return 0;
    const uint64_t cap = CAP - nbins;
    return (nR + 31) / 32 + 1 <= cap * DIRECT_PARTS ? (uint32_t)cap : 0u;
}

// The same for the payload table of a materialising join: 16 entries per row,
// at most 2^24 entries (67 MB).  Measured on 2^28 S rows, gather and 12 B rows
// out: 2.2 ms for tables up to 17 MB, 4.3 ms at 67 MB, 5.6 ms at 134 MB; the
// partitioned join takes about 5 ms.
int direct_log2_max_rows(uint64_t nR) {
    int k = DIRECT_MIN_LOG2;
    while (k < 24 && (1ull << k) < nR * 16) k++;
    return k;
}

// Clears the control block (CTA 0) and, when a sample of R allows a direct
// join, the table (bits to 0, payloads to the empty mark).  Every CTA takes the same 1024 evenly spaced rows, so
// all come to the same w: the sample's range plus 1/32 (evenly spaced rows of
// a relation in random or sorted order miss about 1/1024 of it at either end;
// a range that is wider after all only means "not direct").  More rows than
// the table has entries cannot be distinct.
__global__ void __launch_bounds__(DIRECT_THREADS) k_direct_prep(const Row *__restrict__ R, uint64_t nR,
                                                                uint32_t *__restrict__ table, int log2_max,
                                                                bool payloads, Ctrl *ctrl) {
    __shared__ uint32_t s_lo, s_hi;
    const int tid = threadIdx.x;
    if (blockIdx.x == 0)
        for (int i = tid; i < (int)(sizeof(Ctrl) / 4); i += DIRECT_THREADS) reinterpret_cast<uint32_t *>(ctrl)[i] = 0;
    if (tid == 0) {
        s_lo = 0xFFFFFFFFu;
        s_hi = 0;
    }
    __syncthreads();
    const uint64_t i = nR <= DIRECT_THREADS ? tid : (uint64_t)tid * (nR - 1) / (DIRECT_THREADS - 1);
    uint32_t lo = 0xFFFFFFFFu, hi = 0;
    if (i < nR) lo = hi = R[i].key;
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((tid & 31) == 0) {
        atomicMin(&s_lo, lo);
        atomicMax(&s_hi, hi);
    }
    __syncthreads();
    const uint32_t span = s_hi - s_lo;
    const uint64_t want = (uint64_t)span + span / 32 + 64;
    const int w = max(DIRECT_MIN_LOG2, 64 - __clzll((long long)(want - 1)));
    if (w > log2_max || nR > (1ull << w)) return;
    if (blockIdx.x == 0 && tid == 0) ctrl->direct_log2 = (unsigned)w;
    uint4 *b4 = reinterpret_cast<uint4 *>(table);
    const uint64_t n4 = 1ull << (payloads ? w - 2 : w - 7);
    const uint32_t fill = payloads ? EMPTY_PAYLOAD : 0u;
    for (uint64_t q = (uint64_t)blockIdx.x * DIRECT_THREADS + tid; q < n4; q += (uint64_t)gridDim.x * DIRECT_THREADS)
        b4[q] = make_uint4(fill, fill, fill, fill);
}

// Streams rows [lo, hi) of `in` in rounds of 8 rows per thread: fn(x, ok)
// with four row pairs and their validity, warp-uniform trip counts; edge(row)
// for the rows outside the 16-byte aligned body (thread 0).
template <class Fn, class Edge>
__device__ __forceinline__ void stream_pairs(const Row *__restrict__ in, uint64_t lo, uint64_t hi, Fn fn, Edge edge) {
    if (lo >= hi) return;
    const uint64_t head = ((reinterpret_cast<uintptr_t>(in + lo) & 15) != 0) ? 1 : 0;
    const uint64_t body = hi - lo - head;
    const uint32_t nv = (uint32_t)(body / 2);
    const uint4 *v = reinterpret_cast<const uint4 *>(in + lo + head);
    for (uint32_t base = 0; base < nv; base += DIRECT_THREADS * 4) {
        uint4 x[4];
        bool ok[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t i = base + u * DIRECT_THREADS + threadIdx.x;
            ok[u] = i < nv;
            x[u] = ok[u] ? ldg_stream(v + i) : make_uint4(0, 0, 0, 0);
        }
        fn(x, ok);
    }
    if (threadIdx.x == 0) {
        if (head) edge(in[lo]);
        if (body & 1) edge(in[hi - 1]);
    }
}

__device__ __forceinline__ void hist_pairs(uint32_t *sh, const RadixF &rf, const uint4 (&x)[4], const bool (&ok)[4]) {
    const bool dup = warp_has_dups(radix_f(rf, x[0].x), ok[0]);
#pragma unroll
    for (int u = 0; u < 4; u++) {
        hist_add_warp(sh, radix_f(rf, x[u].x), ok[u], dup);
        hist_add_warp(sh, radix_f(rf, x[u].z), ok[u], dup);
    }
}

// R: chunk histograms, key range, bits.  Three things end the attempt before
// all of R is entered; the CTA that sees one tells the grid through
// ctrl->direct_dup, which every CTA looks at once a round (PAYLOADS: every warp,
// with its exchanges):
//   - two equal keys among a warp's neighbouring rows (no atomic needed), which
//     shows sorted and hot keys before they queue at one word: 2^22 x 2^23 rows,
//     R's last quarter one key, RSM 0.52 ms against 1.18;
//   - a key already there in a careful round, whose atomics return: a sixteenth
//     of the rounds of long chunks, else one round of every sixteenth chunk;
//   - a payload already there (PAYLOADS: every row exchanges its payload with
//     the key's entry, 2^22 rows: 37 us).
// The other rows use atomics without a result, and a duplicate there shows in
// the count of set bits.  Bound by the L2's atomics: 2^27 rows take 0.80 ms
// without results against 1.17 ms with; the histogram read alone 0.16 ms.
template <bool PAYLOADS>
__global__ void __launch_bounds__(DIRECT_THREADS, 2) k_hist_build(const Row *__restrict__ in, uint64_t n, uint64_t chunk,
                                                                  uint32_t *__restrict__ hist, int nbins, RadixF rf,
                                                                  uint32_t *__restrict__ table, Ctrl *ctrl, uint32_t first) {
    dep_wait();
    dep_trigger();
    extern __shared__ uint32_t sh[];
    __shared__ uint32_t s_inv, s_hi;
    __shared__ volatile unsigned s_off;  // as *gave_up of an earlier round
    const int tid = threadIdx.x;
    for (int i = tid; i < nbins; i += DIRECT_THREADS) sh[i] = 0;
    if (tid == 0) s_inv = s_hi = s_off = 0;
    __syncthreads();
    const unsigned w = ctrl->direct_log2;
    const uint32_t wmask = w ? (uint32_t)((1ull << w) - 1) : 0u;
    const uint32_t c = first + blockIdx.x;  // this CTA's chunk
    const uint64_t lo = (uint64_t)c * chunk;
    const uint64_t hi = umin64(n, lo + chunk);
    volatile unsigned *gave_up = &ctrl->direct_dup;
    bool enter = w != 0;  // the same for all lanes of a warp
    uint32_t kinv = 0, kmax = 0;  // largest ~key (the smallest key) and largest key
    // a sixteenth of the rounds of long chunks, of the chunks when they are short
    const uint32_t rounds16 = (uint32_t)(chunk / (16 * 8 * DIRECT_THREADS));
    const uint32_t careful = PAYLOADS ? 0xFFFFFFFFu : rounds16 ? rounds16 : (c & 15) == 0 ? 1u : 0u;
    uint32_t round = 0;
    // enters a row; with ret, true says that the join is not direct
    auto set_bit = [&](uint32_t key, uint32_t payload, bool ret) {
        const uint32_t s = key & wmask;
        kinv = max(kinv, ~key);
        kmax = max(kmax, key);
        if (PAYLOADS) return atomicExch(table + s, payload) != EMPTY_PAYLOAD || payload == EMPTY_PAYLOAD;
        if (!ret) {
            atomicOr(table + (s >> 5), 1u << (s & 31));
            return false;
        }
        return ((atomicOr(table + (s >> 5), 1u << (s & 31)) >> (s & 31)) & 1u) != 0;
    };
    stream_pairs(
        in, lo, hi,
        [&](const uint4(&x)[4], const bool(&ok)[4]) {
            if (enter) {
                if (!PAYLOADS && tid == 0 && round && *gave_up) s_off = 1;
                // rows side by side (u), or in the next lane's pair, with one key
                bool same = s_off != 0;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t before = __shfl_up_sync(0xffffffffu, x[u].z, 1);
                    same |= ok[u] && (x[u].x == x[u].z || (x[u].x == before && (tid & 31) != 0));
                }
                enter = !__any_sync(0xffffffffu, same);
                if (!enter && (tid & 31) == 0 && !*gave_up) *gave_up = 1;
            }
            if (enter) {
                if (round < careful) {
                    bool dup = false;
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        if (ok[u]) {
                            dup |= set_bit(x[u].x, x[u].y, true);
                            dup |= set_bit(x[u].z, x[u].w, true);
                        }
                    }
                    // one lane per warp touches the flag: all of them storing
                    // it took 0.5 ms from a 2^22 x 2^24 join with triplicate keys
                    dup = __any_sync(0xffffffffu, dup);
                    unsigned seen = 0;
                    if ((tid & 31) == 0) {
                        seen = *gave_up;
                        if (dup && !seen) *gave_up = 1;
                    }
                    enter = !dup && __shfl_sync(0xffffffffu, seen, 0) == 0;
                } else {
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        if (ok[u]) {
                            set_bit(x[u].x, x[u].y, false);
                            set_bit(x[u].z, x[u].w, false);
                        }
                    }
                }
                round++;
            }
            __syncwarp();
            hist_pairs(sh, rf, x, ok);
        },
        [&](const Row &r) {
            if (enter && set_bit(r.key, r.payload, false)) *gave_up = 1;
            atomicAdd(&sh[radix_f(rf, r.key)], 1u);
        });
    if (w) {
        for (int o = 16; o > 0; o >>= 1) {
            kinv = max(kinv, __shfl_xor_sync(0xffffffffu, kinv, o));
            kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
        }
        if ((tid & 31) == 0) {
            atomicMax(&s_inv, kinv);
            atomicMax(&s_hi, kmax);
        }
    }
    __syncthreads();
    if (w && tid == 0 && lo < hi) {
        atomicMax(&ctrl->direct_inv_min, s_inv);
        atomicMax(&ctrl->direct_max, s_hi);
    }
    uint32_t *dst = hist + (uint64_t)c * nbins;
    for (int i = tid; i < nbins; i += DIRECT_THREADS) dst[i] = sh[i];
}

// Counts the set bits; the last CTA decides.  The table is read from L2
// (2^27 keys: 33.5 MB, half of it R's range).  A payload table (null bits)
// needs no count: its entries showed every duplicate.  CTA 0 also looks at 1024
// evenly spaced rows of S (null: not there yet) for hot keys: under Zipf z = 1
// over 16.8 M keys they hold thousands of equal pairs, uniform keys hardly any.
__global__ void __launch_bounds__(DIRECT_THREADS) k_direct_decide(const uint32_t *__restrict__ bits, uint64_t nR,
                                                                  const Row *__restrict__ S, uint64_t nS, Ctrl *ctrl) {
    dep_wait();
    dep_trigger();
    __shared__ unsigned s_count;
    const unsigned w = ctrl->direct_log2;
    if (!w || ctrl->direct_dup) return;
    const int tid = threadIdx.x;
    if (!bits) {
        if (blockIdx.x == 0 && tid == 0 && (uint64_t)(ctrl->direct_max - ~ctrl->direct_inv_min) < (1ull << w))
            ctrl->direct = 1;
        return;
    }
    if (tid == 0) s_count = 0;
    if (blockIdx.x == 0) {
        __shared__ uint32_t seen[4096];  // a sampled key at its hash: the later of two keys stays
        __shared__ unsigned equal;
        if (tid == 0) equal = 0;
        for (int i = tid; i < 4096; i += DIRECT_THREADS) seen[i] = ~0u;
        __syncthreads();
        if (S && (uint64_t)tid < nS) {
            const uint64_t i = nS <= DIRECT_THREADS ? tid : (uint64_t)tid * (nS - 1) / (DIRECT_THREADS - 1);
            const uint32_t k = S[i].key;
            if (k != ~0u && atomicExch(&seen[(k * 0x9E3779B1u) >> 20], k) == k) atomicAdd(&equal, 1u);
        }
        __syncthreads();
        if (tid == 0) ctrl->direct_hot = !S || equal >= 16;
    }
    __syncthreads();
    const uint4 *b4 = reinterpret_cast<const uint4 *>(bits);
    const uint64_t n4 = 1ull << (w - 7);
    unsigned c = 0;  // at most 2^29 bits in all
#pragma unroll 4
    for (uint64_t q = (uint64_t)blockIdx.x * DIRECT_THREADS + tid; q < n4; q += (uint64_t)gridDim.x * DIRECT_THREADS) {
        const uint4 x = __ldcg(b4 + q);
        c += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((tid & 31) == 0 && c) atomicAdd(&s_count, c);
    __syncthreads();
    if (tid == 0) {
        atomicAdd(&ctrl->direct_bits, (unsigned long long)s_count);
        __threadfence();
        if (atomicAdd(&ctrl->done[3], 1u) == gridDim.x - 1) {
            __threadfence();
            const unsigned long long set = atomicAdd(&ctrl->direct_bits, 0ull);
            if (set == nR && (uint64_t)(ctrl->direct_max - ~ctrl->direct_inv_min) < (1ull << w)) ctrl->direct = 1;
        }
    }
}

// S: chunk histograms and, when the join is direct, the matches.  Two
// launches, of which one does the work: k_hist_probe_smem reads the table from
// shared memory when it fits there, in up to DIRECT_PARTS parts; k_hist_probe
// reads it from L2, and is the plain histogram when the join is not direct.
// (One launch for both would hold the copy's shared memory, and so one CTA per
// SM, for the plain histogram too: a sparse 2^20 x 2^22 join took 182 us
// instead of 140 us.)

// The words of the table that R's range covers: first word, number of words.
__device__ __forceinline__ uint2 direct_words(const Ctrl *ctrl) {
    const uint32_t kmin = ~ctrl->direct_inv_min, kmax = ctrl->direct_max;
    return make_uint2(kmin >> 5, (kmax >> 5) - (kmin >> 5) + 1);
}
// Whether they fit the copies of at most `parts_max` CTAs.
__device__ __forceinline__ bool direct_fits(uint32_t words, uint32_t smem_words, uint32_t parts_max) {
    return words <= (uint64_t)smem_words * parts_max;
}

// The table in L2: bound by the L1's one line per clock and SM (2^30 rows 4.13
// ms, 8 B/row: 2.1 TB/s; 4.02 ms without the histogram).  The partitioned join
// reads and writes 40 more bytes per row of S.
__global__ void __launch_bounds__(DIRECT_THREADS, 2)
    k_hist_probe(const Row *__restrict__ in, uint64_t n, uint64_t chunk, uint32_t *__restrict__ hist, int nbins, RadixF rf,
                 const uint32_t *__restrict__ bits, uint32_t smem_words, uint32_t parts_max, Ctrl *ctrl) {
    dep_wait();
    dep_trigger();
    const bool direct = ctrl->direct != 0;
    const uint32_t kmin = ~ctrl->direct_inv_min, span = ctrl->direct_max - kmin;
    const uint32_t wordmask = direct ? (uint32_t)((1ull << (ctrl->direct_log2 - 5)) - 1) : 0u;
    if (direct && direct_fits(direct_words(ctrl).y, smem_words, parts_max)) return;
    extern __shared__ uint32_t sh[];
    const int tid = threadIdx.x;
    for (int i = tid; i < nbins; i += DIRECT_THREADS) sh[i] = 0;
    __syncthreads();
    const uint64_t lo = (uint64_t)blockIdx.x * chunk;
    const uint64_t hi = umin64(n, lo + chunk);
    uint32_t matches = 0;  // a chunk holds < 2^32 rows, and a row matches at most once
    auto bit = [](uint32_t word, uint32_t key) { return (word >> (key & 31)) & 1u; };
    auto probe = [&](auto load) {
        auto word = [&](uint32_t key, bool ok) -> uint32_t {
            return ok && key - kmin <= span ? load(bits + ((key >> 5) & wordmask)) : 0u;
        };
        stream_pairs(
            in, lo, hi,
            [&](const uint4(&x)[4], const bool(&ok)[4]) {
                uint32_t a[8];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    a[2 * u] = word(x[u].x, ok[u]);
                    a[2 * u + 1] = word(x[u].z, ok[u]);
                }
                hist_pairs(sh, rf, x, ok);  // while the words arrive
#pragma unroll
                for (int u = 0; u < 4; u++) matches += bit(a[2 * u], x[u].x) + bit(a[2 * u + 1], x[u].z);
            },
            [&](const Row &r) {
                matches += bit(word(r.key, true), r.key);
                atomicAdd(&sh[radix_f(rf, r.key)], 1u);
            });
    };
    // Through the L1, hot keys are found there instead of queueing at their L2
    // slice (16.8 M x 134 M rows, Zipf z = 1: 0.53 against 1.50 ms past it; z =
    // 1.5: 0.43 against 2.18 ms).  Uniform keys gain from it in tables up to 4
    // MB (9%) and above 28 MB, which crowd the L2 (5% at 34 MB, 18% at 67), and lose 2.5%
    // between.
    const uint32_t bytes = span / 8;
    if (!direct) {
        stream_pairs(
            in, lo, hi, [&](const uint4(&x)[4], const bool(&ok)[4]) { hist_pairs(sh, rf, x, ok); },
            [&](const Row &r) { atomicAdd(&sh[radix_f(rf, r.key)], 1u); });
    } else if (ctrl->direct_hot || bytes <= (4u << 20) || bytes > (28u << 20)) {
        probe([](const uint32_t *p) { return __ldg(p); });
    } else {
        probe([](const uint32_t *p) { return ldg_no_l1(p); });
    }
    if (direct) {
        const unsigned long long ws = warp_sum_u64(matches);
        if ((tid & 31) == 0 && ws) atomicAdd(&ctrl->matches, ws);
    }
    __syncthreads();
    uint32_t *dst = hist + (uint64_t)blockIdx.x * nbins;
    for (int i = tid; i < nbins; i += DIRECT_THREADS) dst[i] = sh[i];
}

// The table in shared memory: CTA b holds part b mod `parts` of it and, with
// the other CTAs of its part, reads all of S in rounds of 8192 rows; round u is
// counted in the histogram by the part u mod `parts`.  A direct join uses the
// histograms' column sums only, so a CTA's counts go to row b of the G rows
// whatever chunks they are from, and it clears the rows b + gridDim, ....
// 1.8 M x 36 M rows (two parts): 186 us against 270 us from L2.
__global__ void __launch_bounds__(DIRECT_THREADS, 1)
    k_hist_probe_smem(const Row *__restrict__ in, uint64_t n, int G, uint32_t *__restrict__ hist, int nbins, RadixF rf,
                      const uint32_t *__restrict__ bits, uint32_t smem_words, uint32_t parts_max, Ctrl *ctrl) {
    dep_wait();
    dep_trigger();
    constexpr uint32_t T = DIRECT_THREADS;
    if (!ctrl->direct) return;
    const uint2 all = direct_words(ctrl);
    if (!direct_fits(all.y, smem_words, parts_max)) return;
    extern __shared__ uint32_t sh[];
    uint32_t *copy = sh + nbins;
    const int tid = threadIdx.x;
    const uint32_t parts = (all.y + smem_words - 1) / smem_words;  // <= parts_max <= gridDim.x
    const uint32_t per = (all.y + parts - 1) / parts;              // <= smem_words
    const uint32_t part = blockIdx.x % parts, member = blockIdx.x / parts;
    const uint32_t members = (gridDim.x - part + parts - 1) / parts;
    const uint32_t wordmask = (uint32_t)((1ull << (ctrl->direct_log2 - 5)) - 1);
    const uint32_t w0 = all.x + min(part * per, all.y), words = min(per, all.x + all.y - w0);
    // this part's keys: [klo, klo + kspan] (kspan: none for a part past the end)
    const uint32_t kmin = ~ctrl->direct_inv_min, kmax = ctrl->direct_max;
    const uint32_t klo = max(kmin, w0 << 5), khi = min(kmax, ((w0 + words - 1) << 5) | 31);
    const bool none = words == 0;
    const uint32_t kspan = none ? 0 : khi - klo;
    for (int i = tid; i < nbins; i += T) sh[i] = 0;
    for (uint32_t i = tid; i < words; i += T) copy[i] = __ldg(bits + ((w0 + i) & wordmask));
    __syncthreads();
    uint32_t matches = 0;  // this thread's: at most one per row
    auto look = [&](uint32_t key) {
        if (key - klo <= kspan && !none) matches += (copy[(key >> 5) - w0] >> (key & 31)) & 1u;
    };
    const uint32_t head = (reinterpret_cast<uintptr_t>(in) & 15) ? 1u : 0u;
    const uint32_t nv = (uint32_t)((n - head) / 2);  // n >= 1
    const uint4 *v = reinterpret_cast<const uint4 *>(in + head);
    uint4 nx[4];
    auto load = [&](uint64_t round) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint64_t i = round * (4 * T) + u * T + tid;
            nx[u] = i < nv ? ldg_stream(v + i) : make_uint4(0, 0, 0, 0);
        }
    };
    load(member);
    for (uint64_t round = member; round * (4 * T) < nv; round += members) {
        uint4 x[4];
        bool ok[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            x[u] = nx[u];
            ok[u] = round * (4 * T) + u * T + tid < nv;
        }
        load(round + members);  // in flight during this round
        if (round % parts == part) hist_pairs(sh, rf, x, ok);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (ok[u]) {
                look(x[u].x);
                look(x[u].z);
            }
        }
    }
    if (member == 0 && tid == 0) {  // the rows outside the 16-byte aligned body
        auto edge = [&](uint32_t key) {
            look(key);
            if (part == 0) atomicAdd(&sh[radix_f(rf, key)], 1u);
        };
        if (head) edge(in[0].key);
        if ((n - head) & 1) edge(in[n - 1].key);
    }
    const unsigned long long ws = warp_sum_u64(matches);
    if ((tid & 31) == 0 && ws) atomicAdd(&ctrl->matches, ws);
    __syncthreads();
    for (int c = blockIdx.x; c < G; c += gridDim.x) {
        uint32_t *dst = hist + (uint64_t)c * nbins;
        const bool mine = c == (int)blockIdx.x;
        for (int i = tid; i < nbins; i += T) dst[i] = mine ? sh[i] : 0u;
    }
}

// S of a materialising join: chunk histograms and, when the join is direct,
// the output rows.  A round takes 8 rows per thread: their payloads are
// gathered from the table in L2, the matching rows take places in (warp, row
// slot, lane) order in shared memory, and one atomic reserves the round's
// output.  A round's rows leave for memory while the next round's payloads
// arrive, and the reservation returns while the rows are staged, so a round
// waits for neither.  Bound by L2 (one sector per row gathered, 12 B out, 8 B
// in): 16.8 M rows take 128 us, 161 us before the rounds overlapped (then
// with a bulk store per round); as a relation (REL) 120 us.
constexpr int EMIT_DIRECT_THREADS = 512;
constexpr int EMIT_ROUND = EMIT_DIRECT_THREADS * 8;

struct EmitSmem {
    alignas(16) uint32_t stage[EMIT_ROUND * 3];
    uint32_t wtot[EMIT_DIRECT_THREADS / 32];
    unsigned long long base;
};

// REL: the output is a relation of (key, R payload) tuples, what a chained join
// makes of the rows (chain.cu): 8 B a row, and no conversion afterwards.
template <bool REL>
__global__ void __launch_bounds__(EMIT_DIRECT_THREADS, 2)
    k_hist_emit(const Row *__restrict__ in, uint64_t n, uint64_t chunk, uint32_t *__restrict__ hist, int nbins, RadixF rf,
                const uint32_t *__restrict__ table, uint32_t *__restrict__ out, uint64_t cap, uint32_t range_max,
                Ctrl *ctrl) {
    constexpr uint32_t W = REL ? 2 : 3;  // words per output row
    dep_wait();
    dep_trigger();
    constexpr int T = EMIT_DIRECT_THREADS, NW = T / 32;
    extern __shared__ __align__(16) unsigned char esmem[];
    EmitSmem &sm = *reinterpret_cast<EmitSmem *>(esmem);
    uint32_t *sh = reinterpret_cast<uint32_t *>(esmem + sizeof(EmitSmem));
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int i = tid; i < nbins; i += T) sh[i] = 0;
    const bool direct = ctrl->direct != 0;
    const uint32_t kmin = ~ctrl->direct_inv_min, span = ctrl->direct_max - kmin;
    const uint32_t mask = direct ? (uint32_t)((1ull << ctrl->direct_log2) - 1) : 0u;
    __syncthreads();
    const uint64_t lo = (uint64_t)blockIdx.x * chunk;
    const uint64_t hi = umin64(n, lo + chunk);
    unsigned long long matches = 0;  // not direct: keys outside range_max
    uint32_t staged = 0;             // rows of the last round in the stage, at sm.base
    // writes the staged rows out, word by word (coalesced)
    auto flush = [&]() {
        const unsigned long long base = sm.base;
        const uint32_t words = base < cap ? W * (uint32_t)umin64(staged, cap - base) : 0u;
        uint32_t *g = out + base * W;
#pragma unroll 4
        for (uint32_t i = tid; i < words; i += T) __stcs(g + i, sm.stage[i]);
    };
    // one round: this thread's rows (k, p) of `valid`; every thread calls it
    auto round = [&](const uint32_t (&k)[8], const uint32_t (&p)[8], unsigned valid) {
        uint32_t r[8];
        if (direct) {
#pragma unroll
            for (int j = 0; j < 8; j++)
                r[j] = (valid >> j & 1) && k[j] - kmin <= span ? __ldg(table + (k[j] & mask)) : EMPTY_PAYLOAD;
            flush();  // the last round's rows, while the payloads arrive
        }
        const bool dup = warp_has_dups(radix_f(rf, k[0]), valid & 1u);
#pragma unroll
        for (int j = 0; j < 8; j++) hist_add_warp(sh, radix_f(rf, k[j]), valid >> j & 1, dup);
        if (!direct) {
            if (range_max != 0xFFFFFFFFu) {  // as k_hist_chunks: keys outside the bins' range
                unsigned o = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) o += (valid >> j & 1) && k[j] - rf.sub > range_max;
                matches += o;
            }
            return;
        }
        unsigned m[8], wt = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            m[j] = __ballot_sync(0xffffffffu, r[j] != EMPTY_PAYLOAD);
            wt += __popc(m[j]);
        }
        if (lane == 0) sm.wtot[w] = wt;
        __syncthreads();  // totals written, the stage free
        uint32_t before = 0, total = 0;
#pragma unroll
        for (int q = 0; q < NW; q++) {
            const uint32_t x = sm.wtot[q];
            before += q < w ? x : 0;
            total += x;
        }
        unsigned long long base = 0;
        if (tid == 0 && total) base = atomicAdd(&ctrl->rows, (unsigned long long)total);
        const unsigned lt = lanemask_lt();
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (m[j] >> lane & 1) {
                uint32_t *q = sm.stage + W * (before + __popc(m[j] & lt));
                q[0] = k[j];
                q[1] = r[j];
                if (!REL) q[2] = p[j];
            }
            before += __popc(m[j]);
        }
        if (tid == 0) {
            sm.base = base;
            matches += total;
        }
        staged = total;
        __syncthreads();  // staged, and its place known
    };
    if (lo < hi) {
        const uint32_t head = ((reinterpret_cast<uintptr_t>(in + lo) & 15) != 0) ? 1 : 0;
        const uint64_t body = hi - lo - head;
        const uint32_t nv = (uint32_t)(body / 2);
        const bool tail = body & 1;
        const uint4 *v = reinterpret_cast<const uint4 *>(in + lo + head);
        uint4 nx[4];
        auto load_round = [&](uint32_t b) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint32_t i = b + u * T + tid;
                nx[u] = i < nv ? ldg_stream(v + i) : make_uint4(0, 0, 0, 0);
            }
        };
        load_round(0);
        for (uint32_t b = 0; b < nv; b += 4 * T) {
            uint32_t k[8], p[8];
            unsigned valid = 0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                k[2 * u] = nx[u].x;
                p[2 * u] = nx[u].y;
                k[2 * u + 1] = nx[u].z;
                p[2 * u + 1] = nx[u].w;
                if (b + u * T + tid < nv) valid |= 3u << (2 * u);
            }
            load_round(b + 4 * T);  // in flight during this round
            round(k, p, valid);
        }
        if (head || tail) {  // the edge rows: one round of at most two rows
            uint32_t k[8] = {}, p[8] = {};
            unsigned valid = 0;
            if ((tid == 0 && head) || (tid == 1 && tail)) {
                const Row r = in[tid == 0 ? lo : hi - 1];
                k[0] = r.key;
                p[0] = r.payload;
                valid = 1;
            }
            round(k, p, valid);
        }
        if (direct) flush();
    }
    if (direct) {  // thread 0 counted the rounds' rows
        if (tid == 0 && matches) atomicAdd(&ctrl->matches, matches);
    } else {
        const unsigned long long o = warp_sum_u64(matches);
        if (lane == 0 && o) atomicAdd(&ctrl->out_of_range, o);
    }
    __syncthreads();
    uint32_t *hdst = hist + (uint64_t)blockIdx.x * nbins;
    for (int i = tid; i < nbins; i += T) hdst[i] = sh[i];
}

cudaError_t launch_hist_emit(const Row *in, uint64_t n, uint64_t chunk, int G, uint32_t *hist, int P_log2, RadixF rf,
                             const uint32_t *table, tbg_row_out *out, Row *rel, uint64_t cap, uint32_t range_max, Ctrl *ctrl,
                             cudaStream_t st) {
    const int nbins = 1 << P_log2;
    const size_t smem = sizeof(EmitSmem) + (size_t)nbins * 4;
    auto kern = rel ? k_hist_emit<true> : k_hist_emit<false>;
    uint32_t *words = rel ? reinterpret_cast<uint32_t *>(rel) : reinterpret_cast<uint32_t *>(out);
    cudaError_t e = smem_limit((const void *)kern, smem);
    if (e != cudaSuccess) return e;
    e = launch_dep(kern, G, EMIT_DIRECT_THREADS, smem, st, in, n, chunk, hist, nbins, rf, table, words, cap, range_max, ctrl);
    count_launch();
    return e;
}

cudaError_t launch_direct_prep(const Row *R, uint64_t nR, uint32_t *table, int log2_max, bool payloads, Ctrl *ctrl,
                               int nsm, cudaStream_t st) {
    const uint64_t n4 = 1ull << (payloads ? log2_max - 2 : log2_max - 7);
    const unsigned g = (unsigned)std::min<uint64_t>((n4 + DIRECT_THREADS - 1) / DIRECT_THREADS, (uint64_t)nsm * 2);
    k_direct_prep<<<g, DIRECT_THREADS, 0, st>>>(R, nR, table, log2_max, payloads, ctrl);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_hist_build(const Row *in, uint64_t n, uint64_t chunk, int G, uint32_t *hist, int P_log2, RadixF rf,
                              uint32_t *table, bool payloads, int wave, Ctrl *ctrl, cudaStream_t st) {
    const int nbins = 1 << P_log2;
    const size_t smem = (size_t)nbins * 4;
    auto kern = payloads ? k_hist_build<true> : k_hist_build<false>;
    cudaError_t e = smem_limit((const void *)kern, smem);
    if (e != cudaSuccess) return e;
    if (!wave || wave >= G) {
        e = launch_dep(kern, G, DIRECT_THREADS, smem, st, in, n, chunk, hist, nbins, rf, table, ctrl, 0u);
        count_launch();
        return e;
    }
    // plain launches: a dependent one's CTAs would take the room that the
    // waves are there to leave
    for (int c = 0; c < G; c += wave) {
        kern<<<std::min(wave, G - c), DIRECT_THREADS, smem, st>>>(in, n, chunk, hist, nbins, rf, table, ctrl, (uint32_t)c);
        count_launch();
    }
    return cudaGetLastError();
}

cudaError_t launch_direct_decide(const uint32_t *bits, int log2_max, uint64_t nR, const Row *S, uint64_t nS, int wave, int nsm,
                                 Ctrl *ctrl, cudaStream_t st) {
    const uint64_t n4 = 1ull << (log2_max - 7);
    // two 16-byte words per thread and CTA at least, one CTA per SM at most
    const unsigned g = bits ? (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(n4 / (DIRECT_THREADS * 2), (uint64_t)nsm)) : 1u;
    if (wave) {  // no dependent launch, as above
        k_direct_decide<<<g, DIRECT_THREADS, 0, st>>>(bits, nR, S, nS, ctrl);
        count_launch();
        return cudaGetLastError();
    }
    const cudaError_t e = launch_dep(k_direct_decide, g, DIRECT_THREADS, 0, st, bits, nR, S, nS, ctrl);
    count_launch();
    return e;
}

cudaError_t launch_hist_probe(const Row *in, uint64_t n, uint64_t chunk, int G, uint32_t *hist, int P_log2, RadixF rf,
                              const uint32_t *bits, uint64_t nR, int nsm, Ctrl *ctrl, cudaStream_t st) {
    const int nbins = 1 << P_log2;
    const uint32_t words = direct_smem_words(nR, (uint64_t)nbins);
    const unsigned grid = (unsigned)std::min(G, nsm);  // every CTA writes a row of the histogram
    const uint32_t parts_max = std::min<uint32_t>(DIRECT_PARTS, grid);
    const size_t smem = (size_t)nbins * 4, smem_copy = smem + (size_t)words * 4;
    cudaError_t e;
    if (words) {
        if ((e = smem_limit((const void *)k_hist_probe_smem, smem_copy)) != cudaSuccess) return e;
        e = launch_dep(k_hist_probe_smem, grid, DIRECT_THREADS, smem_copy, st, in, n, G, hist, nbins, rf, bits, words,
                       parts_max, ctrl);
        count_launch();
        if (e != cudaSuccess) return e;
    }
    if ((e = smem_limit((const void *)k_hist_probe, smem)) != cudaSuccess) return e;
    e = launch_dep(k_hist_probe, G, DIRECT_THREADS, smem, st, in, n, chunk, hist, nbins, rf, bits, words, parts_max,
                   ctrl);
    count_launch();
    return e;
}

}  // namespace tbg
