// K4: per-partition build/probe out of shared memory, persistent CTAs pulling
// work items.  Replaces the reference's join phase (Joins/radix_join.c:1184-1192
// task loop) and its two table layouts:
//   layout 0  bucket_chaining_join (Joins/radix_join.c:187-244): bucket heads
//             over next_pow2(|R_p|) slots, index (key >> bits) & (N-1),
//             1-based chains through `next`;
//   layout 1  histogram_join (Joins/radix_join.c:374-440, RHT): bucket counts
//             over max(next_pow2(|R_p|)/4, 4) slots, prefix sum, R_p reordered
//             by bucket, probe scans the bucket's range.
// These are the materialising tables.  Counting joins of both layouts build a
// CellTable (join_dev.cuh: 32-bit heads and cells) over partitions of bare keys.
// Counting uses per-thread counters folded once per CTA; materialisation
// reserves output rows once per CTA round (one global atomic for up to
// JOIN_THREADS * 8 probe rows) and places them in (row slot, lane) order, so
// consecutive lanes store consecutive rows (the reference's insert_output,
// Include/util.c:20-29, mallocs one node per row).
#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>

#include "join_dev.cuh"

namespace tbg {

// Heads of a counting table: about one per row (partitions average half the
// table or less, see join_capacity).
__host__ __device__ __forceinline__ uint32_t count_heads(int capR) { return floor_pow2((uint32_t)capR); }

// S keys against a table with long runs (a function of its own, so that the
// plain probe's registers are its own).
__device__ __noinline__ unsigned long long probe_runs(const CellTable t, const uint32_t *s, uint64_t len) {
    return stream_sum<JOIN_THREADS>(s, len, [&](uint32_t k) { return t.count<true>(k); });
}

// Counting: three CTAs per SM (40 registers). Materialising: no bound; the
// compiler takes 64 registers either way, but scheduled for a bound of two CTAs
// it ran 5% slower (2^23 x 2^25 rows that come twice: 524 against 496 us).
template <bool MAT>
__global__ void __launch_bounds__(JOIN_THREADS, MAT ? 0 : 3) k_join(JoinArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_item[2];
    __shared__ uint64_t scan_scratch[JOIN_THREADS / 32 + 1];
    dep_wait();
    dep_trigger();
    if (a.skip && *a.skip) return;
    if (a.gate) {  // the same value for every thread: the whole launch steps aside
        const unsigned long long v = *a.gate;
        if (a.gate_le ? v > a.gate_max : v <= a.gate_max) return;
    }
    Table t;
    CellTable ct;
    __shared__ std::conditional_t<MAT, uint32_t, LongRuns> runs;
    if (MAT) {
        t.key = reinterpret_cast<uint32_t *>(smem);
        t.pay = t.key + a.capR;
        t.heads = t.pay + a.capR;
        t.next = reinterpret_cast<uint16_t *>(t.heads + a.capR + 2);
        t.hcap = floor_pow2((uint32_t)a.capR + 2);
        t.hs = a.hash_shift;
        t.layout = a.layout;
    } else {
        ct.hcap = count_heads(a.capR);
        ct.heads = reinterpret_cast<uint32_t *>(smem);
        ct.cells = ct.heads + ct.hcap;
        ct.hs = a.hash_shift;
        ct.link_bits = cell_link_bits((uint32_t)a.capR);
        ct.runs = reinterpret_cast<LongRuns *>(&runs);
    }
    const int tid = threadIdx.x;
    const unsigned nitems = *a.err ? 0u : *a.nitems;  // a planner error leaves the item list unusable
    unsigned long long local = 0;
    // counting: the partitions hold bare keys
    const uint32_t *Rk = reinterpret_cast<const uint32_t *>(a.R), *Sk = reinterpret_cast<const uint32_t *>(a.S);

    // the next item is claimed when the current one's table is built, and its R
    // rows are prefetched into L2 while the current item is probed, so its table
    // build reads L2.  (Claimed before the build, with few items, CTAs took two
    // while others had none: 2^20 x 2^20 rows, 128 items, 31 us against 24.)
    if (tid == 0) s_item[0] = atomicAdd(a.item_ctr, 1u);
    __syncthreads();
    for (uint32_t iter = 0;; iter++) {
        const uint32_t it = s_item[iter & 1];
        if (it >= nitems) break;
        if (MAT) build_table<JOIN_THREADS>(t, a.R, a.items[it].r_off, a.items[it].r_len, scan_scratch);
        else build_cells<JOIN_THREADS, false, RUNS_CALL>(ct, Rk, a.items[it].r_off, a.items[it].r_len);
        if (tid == 0) {
            const uint32_t nx = atomicAdd(a.item_ctr, 1u);
            s_item[(iter + 1) & 1] = nx;  // read by all after this item's barriers
            if (nx < nitems) {
                const Item mn = a.items[nx];
                if (MAT) prefetch_l2(a.R + mn.r_off, (uint64_t)mn.r_len * sizeof(Row));
                else prefetch_l2(Rk + mn.r_off, (uint64_t)mn.r_len * 4);
            }
        }

        const uint64_t s_off = a.items[it].s_off, len = a.items[it].s_len;
        const Row *s = a.S + s_off;
        const uint64_t head = ((reinterpret_cast<uintptr_t>(s) & 15) && len) ? 1 : 0;
        const uint64_t body = len - head;
        const uint64_t nv = body / 2;
        const bool tail = body & 1;
        const uint4 *v = reinterpret_cast<const uint4 *>(s + head);

        if (!MAT) {
            if (!ct.has_runs) local += probe_count<JOIN_THREADS>(ct, Sk + s_off, len);
            else local += probe_runs(ct, Sk + s_off, len);
        } else {
            // block-synchronous rounds: 8 rows per thread, one reservation per round
            const uint64_t per_round = 4ull * JOIN_THREADS;
            const uint64_t rounds = (nv + per_round - 1) / per_round + ((head || tail) ? 1 : 0);
            for (uint64_t r = 0; r < rounds; r++) {
                uint32_t k[8], p[8];
                unsigned valid = 0;
                const bool edge = (head || tail) && r == rounds - 1;
                if (edge) {
                    if (tid == 0 && head) { k[0] = s[0].key; p[0] = s[0].payload; valid = 1; }
                    if (tid == 1 && tail) { k[0] = s[len - 1].key; p[0] = s[len - 1].payload; valid = 1; }
                } else {
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        uint64_t i = r * per_round + (uint64_t)u * JOIN_THREADS + tid;
                        if (i < nv) {
                            uint4 x = ldg_stream(v + i);
                            k[2 * u] = x.x; p[2 * u] = x.y;
                            k[2 * u + 1] = x.z; p[2 * u + 1] = x.w;
                            valid |= 3u << (2 * u);
                        }
                    }
                }
                uint32_t c[8];
                uint32_t csum = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    c[j] = (valid >> j & 1) ? t.count(k[j]) : 0;
                    csum += c[j];
                }
                uint64_t pos[8];
                block_emit_positions<JOIN_THREADS, 8>(c, pos, a.rows_ctr, scan_scratch);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (c[j]) {
                        const uint32_t kk = k[j], pp = p[j];
                        uint64_t q = pos[j];
                        t.for_each(kk, [&](uint32_t rp) {
                            if (q < a.cap) {
                                tbg_row_out o;
                                o.key = kk; o.Rpayload = rp; o.Spayload = pp;
                                a.out[q] = o;
                            }
                            q++;
                        });
                    }
                }
                const uint32_t c_total = csum;
                local += c_total;
            }
        }
        __syncthreads();  // table reused by the next item
    }
    unsigned long long ws = warp_sum_u64(local);
    if ((tid & 31) == 0 && ws) atomicAdd(a.matches, ws);
}

size_t join_smem_bytes(int capR) {
    return (size_t)capR * 4 * 2 + ((size_t)capR + 2) * 4 + (size_t)capR * 2 + 16;
}
// Shared memory of a k_join launch (counting: heads and cells).
size_t join_launch_smem(int capR, bool materialize) {
    if (!materialize) return ((size_t)count_heads(capR) + capR) * 4;
    return join_smem_bytes(capR);
}

// Resident CTAs per SM of a k_join launch at a table of capR rows, cached per
// (device, capR, materialize): the occupancy query runs once per size.
int join_ctas_per_sm(int capR, bool materialize) {
    static std::mutex mu;
    static std::map<std::pair<int, int>, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> g(mu);
    const int key = capR * 2 + (materialize ? 1 : 0);
    auto it = cache.find(std::make_pair(dev, key));
    if (it != cache.end()) return it->second;
    const size_t smem = join_launch_smem(capR, materialize);
    int n = 0;
    if (smem_limit((const void *)k_join<false>, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_join<false>, JOIN_THREADS, smem) != cudaSuccess) {
        cudaGetLastError();
        return 1;  // not cached: a later call retries
    }
    n = n < 1 ? 1 : n;
    cache[std::make_pair(dev, key)] = n;
    return n;
}

cudaError_t launch_join(const JoinArgs &a, bool materialize, int grid, cudaStream_t st) {
    const size_t smem = join_launch_smem(a.capR, materialize);
    auto kern = materialize ? k_join<true> : k_join<false>;
    cudaError_t e = smem_limit((const void *)kern, smem);
    if (e != cudaSuccess) return e;
    e = launch_dep(kern, grid, JOIN_THREADS, smem, st, a);
    count_launch();
    return e;
}

}  // namespace tbg
