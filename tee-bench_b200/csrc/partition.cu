// Radix partitioning for sm_100a without inter-CTA waits.
//
// Replaces the reference's two partitioning passes (Joins/radix_join.c:630-703
// parallel_radix_partition, :525-562 radix_cluster, :573-619
// serial_radix_partition, the SWWC variant :734-827) and the task queues that
// feed them (Include/task_queue.h).  The reference's own structure -- every
// thread histograms a contiguous chunk, a prefix over (thread, digit) gives
// each thread exact write cursors, then each thread scatters its chunk -- is
// kept, with a CTA in the role of a thread:
//
//   K1 hist   CTA c histograms chunk c over all final partitions f (2^bits
//             bins in shared memory) -> hist[c][f];
//   K2 scan   column prefix over chunks -> pre[c][f], totals[f];
//   K3 plan   exclusive scan of totals -> base[f], join work items;
//   K4 pass 1 CTA c scatters chunk c by the pass-1 digit d1 = f >> b2 to
//             cursor[d1] = base[d1 << b2] + sum_{d2} pre[c][(d1 << b2) | d2];
//   K5 pass 2 unit (c, s) = the rows chunk c wrote to pass-1 partition s;
//             scattered by d2 to cursor[d2] = base[(s << b2) | d2] + pre[c][...].
//
// One histogram read gives every cursor of both passes, so the traffic is
// 8 (hist) + 16 (pass 1) + 16 (pass 2) bytes per row, and no CTA ever waits
// for another.  A counting join needs no payloads: its pass 1 writes bare keys
// and pass 2 moves those, 8 + 12 + 8 bytes per row.  Each pass stages a tile digit-sorted in shared memory and
// writes runs with consecutive threads on consecutive addresses (coalesced).
#include "part_dev.cuh"

namespace tbg {

// Threads per CTA of the two passes (tiles of THREADS * PART_ITEMS rows).
#ifndef TBG_PASS1_THREADS
#define TBG_PASS1_THREADS 512
#endif
#ifndef TBG_PASS2_THREADS
#define TBG_PASS2_THREADS 512
#endif
constexpr int PASS1_THREADS = TBG_PASS1_THREADS;
constexpr int PASS2_THREADS = TBG_PASS2_THREADS;
// Tile buffers per CTA of the two passes (bulk copies run NBUF - 1 tiles ahead).
#ifndef TBG_PASS_NBUF
#define TBG_PASS_NBUF 3
#endif
constexpr int PASS_NBUF = TBG_PASS_NBUF;
template <int THREADS, class In = Row>
using PassSmem = PartSmem<THREADS, PASS_NBUF, In, sizeof(In) == 8 ? PART_ITEMS : PART_KEY_ITEMS>;

// ---------------------------------------------------------------------------
// K1 per-chunk histogram over the final partition index f
// ---------------------------------------------------------------------------
constexpr int HIST_THREADS = 1024;

// A dependent launch: as a plain one between dependent ones the first pass after
// it took 10 us longer (PSM 2^22 x 2^22, triplicate keys: 195 against 183 us).
// With `oor` set, keys whose key - rf.sub exceeds range_max are also
// counted into *oor (the histogram of a relation binned by another's key
// range: a non-zero count means the bins are not valid).
__global__ void __launch_bounds__(HIST_THREADS) k_hist_chunks(const Row *__restrict__ in, uint64_t n,
                                                             uint64_t chunk, uint32_t *__restrict__ hist,
                                                             int nbins, RadixF rf, unsigned long long *oor,
                                                             uint32_t range_max) {
    dep_wait();
    dep_trigger();
    unsigned outside = 0;
    extern __shared__ uint32_t sh[];
    for (int i = threadIdx.x; i < nbins; i += HIST_THREADS) sh[i] = 0;
    __syncthreads();
    const uint64_t lo = (uint64_t)blockIdx.x * chunk;
    const uint64_t hi = umin64(n, lo + chunk);
    if (lo < hi) {
        const uint64_t head = ((reinterpret_cast<uintptr_t>(in + lo) & 15) != 0) ? 1 : 0;
        const uint64_t body = hi - lo - head;
        const uint64_t nv = body / 2;
        const uint4 *v = reinterpret_cast<const uint4 *>(in + lo + head);
        // warp-uniform trip count: every lane reaches the shuffles
        const uint64_t per = (uint64_t)HIST_THREADS * 4;
        for (uint64_t base = 0; base < nv; base += per) {
            uint4 x[4];
            bool ok[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                uint64_t i = base + (uint64_t)u * HIST_THREADS + threadIdx.x;
                ok[u] = i < nv;
                if (ok[u]) x[u] = ldg_stream(v + i);
            }
            uint32_t f[8];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                f[2 * u] = ok[u] ? radix_f(rf, x[u].x) : 0;
                f[2 * u + 1] = ok[u] ? radix_f(rf, x[u].z) : 0;
                if (oor && ok[u]) outside += (x[u].x - rf.sub > range_max) + (x[u].z - rf.sub > range_max);
            }
            const bool dup = warp_has_dups(f[0], ok[0]);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                hist_add_warp(sh, f[2 * u], ok[u], dup);
                hist_add_warp(sh, f[2 * u + 1], ok[u], dup);
            }
        }
        if (threadIdx.x == 0) {
            if (head) {
                atomicAdd(&sh[radix_f(rf, in[lo].key)], 1u);
                outside += oor && in[lo].key - rf.sub > range_max;
            }
            if (body & 1) {
                atomicAdd(&sh[radix_f(rf, in[hi - 1].key)], 1u);
                outside += oor && in[hi - 1].key - rf.sub > range_max;
            }
        }
    }
    if (oor) {
        const unsigned long long wo = warp_sum_u64((unsigned long long)outside);
        if ((threadIdx.x & 31) == 0 && wo) atomicAdd(oor, wo);
    }
    __syncthreads();
    uint32_t *dst = hist + (uint64_t)blockIdx.x * nbins;
    for (int i = threadIdx.x; i < nbins; i += HIST_THREADS) dst[i] = sh[i];
}

// ---------------------------------------------------------------------------
// K2 column prefix over chunks (in place) and per-partition totals.  A CTA
// owns 32 consecutive partitions (threadIdx.x, coalesced) and splits the
// chunks into 32 segments (threadIdx.y): segment sums, a prefix over the
// segments, then each segment rewritten with running prefixes.
// K3 planner: partition bases and join work items.  Replaces the task
// creation of Joins/radix_join.c:946-1000 and :609-617 (pairs with both sides
// non-empty); oversized S sides are split into several items.
// One launch does K2 for both relations; each relation's last CTA scans its
// bases, and the second of them plans the items: as five launches (two column
// scans, two base scans, the planner) it took 24 us of the 120 us of a
// 2^21 x 2^21 join.
// ---------------------------------------------------------------------------
constexpr int PLAN_THREADS = 1024;

// With totals_only (a direct join, which uses no prefix) the chunks' rows stay
// as they are.
__device__ void column_scan(uint32_t *__restrict__ hist, int G, int P, uint32_t *__restrict__ totals, int block,
                            uint32_t (*seg)[33], bool totals_only) {
    const int f = block * 32 + threadIdx.x;
    const int per = (G + 31) / 32;
    const int c0 = min(G, (int)threadIdx.y * per), c1 = min(G, c0 + per);
    uint32_t *col = hist + f;
    uint32_t sum = 0;
    if (f < P) {
        int c = c0;
        for (; c + 8 <= c1; c += 8) {  // eight independent loads in flight
            uint32_t x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = col[(uint64_t)(c + u) * P];
#pragma unroll
            for (int u = 0; u < 8; u++) sum += x[u];
        }
        for (; c < c1; c++) sum += col[(uint64_t)c * P];
    }
    seg[threadIdx.y][threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.y == 0) {
        uint32_t run = 0;
        for (int y = 0; y < 32; y++) {
            const uint32_t v = seg[y][threadIdx.x];
            seg[y][threadIdx.x] = run;
            run += v;
        }
        if (f < P) totals[f] = run;
    }
    if (totals_only) return;
    __syncthreads();
    if (f < P) {
        uint32_t run = seg[threadIdx.y][threadIdx.x];
        int c = c0;
        for (; c + 8 <= c1; c += 8) {
            uint32_t x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = col[(uint64_t)(c + u) * P];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                col[(uint64_t)(c + u) * P] = run;
                run += x[u];
            }
        }
        for (; c < c1; c++) {
            const uint32_t v = col[(uint64_t)c * P];
            col[(uint64_t)c * P] = run;
            run += v;
        }
    }
}

// Exclusive scan of tot[0..P) into base[0..P], base[P] = total (rows counted:
// n unless rows were bypassed), and the largest entry into *maxp, by one CTA
// of PLAN_THREADS threads.  Warp w owns `per` consecutive entries and walks
// them 32 at a time, so loads and stores are coalesced; up to PLAN_THREADS
// entries that is one load per thread.
__device__ void plan_bases(const uint32_t *tot, uint64_t *base, int P, unsigned long long *maxp, int tid,
                           uint64_t *scratch) {
    const int lane = tid & 31, w = tid >> 5;
    const int per = ((P + 31) / 32 + 31) & ~31;
    const int lo = min(P, w * per), hi = min(P, lo + per);
    const uint32_t first = lo + lane < hi ? __ldcg(tot + lo + lane) : 0;
    uint64_t sum = first;
    uint32_t mx = first;
#pragma unroll 4
    for (int f = lo + 32 + lane; f < hi; f += 32) {
        const uint32_t x = __ldcg(tot + f);
        sum += x;
        mx = max(mx, x);
    }
    sum = warp_sum_u64(sum);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) {
        scratch[w] = sum;
        if (mx) atomicMax(maxp, (unsigned long long)mx);
    }
    __syncthreads();
    const uint64_t ws = scratch[lane];  // 32 warps
    uint64_t winc = ws;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, winc, o);
        if (lane >= o) winc += y;
    }
    uint64_t run = __shfl_sync(0xffffffffu, winc - ws, w);
    const uint64_t total = __shfl_sync(0xffffffffu, winc, 31);
#pragma unroll 4
    for (int f0 = lo; f0 < hi; f0 += 32) {
        const int f = f0 + lane;
        const uint32_t x = f0 == lo ? first : (f < hi ? __ldcg(tot + f) : 0);
        uint32_t inc = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (f < hi) base[f] = run + inc - x;
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (tid == 0) base[P] = total;
    __syncthreads();  // scratch is reused; base is complete for this CTA
}

// Join work items from both relations' totals and bases, for partitions
// block * PLAN_THREADS + tid.  Every call first counts the items of all
// partitions (one coalesced read of both totals, from L2) to take the same
// split decision; each warp then reserves its items with one atomic on
// ctrl->nitems (zeroed before).  The item list is in reservation order, not
// sorted by partition.
__device__ void plan_block(const PlanArgs &a, int block, int tid, uint64_t *scratch) {
    const int P = 1 << a.P_log2;
    // large S sides are split (skew) for every R chunk of the
    // partition; if that would overflow the item buffer, partitions whose R
    // side needs several chunks keep S whole
    auto s_chunks = [&](uint32_t hs, uint64_t nrc, bool split_all) -> uint64_t {
        return nrc > 1 && !split_all ? 1 : a.split.items(hs, nrc);
    };
    const int f = block * PLAN_THREADS + tid;
    const uint32_t hr = f < P ? __ldcg(a.r.hist + f) : 0, hs = f < P ? __ldcg(a.s.hist + f) : 0;
    auto count = [&](uint32_t r, uint32_t s) -> uint64_t {
        if (r == 0 || s == 0) return 0;
        const uint64_t nrc = (r + (uint64_t)a.capR - 1) / a.capR;
        return nrc * s_chunks(s, nrc, true);
    };
    uint64_t cnt_all = count(hr, hs);
    if (P > PLAN_THREADS)
        for (int q = tid; q < P; q += PLAN_THREADS)
            if (q != f) cnt_all += count(__ldcg(a.r.hist + q), __ldcg(a.s.hist + q));
    const int lane = tid & 31, w = tid >> 5;
    cnt_all = warp_sum_u64(cnt_all);
    if (lane == 0) scratch[w] = cnt_all;
    __syncthreads();
    const uint64_t total_all = warp_sum_u64(scratch[lane]);  // 32 warps
    __syncthreads();
    const bool split_all = total_all <= a.item_cap;
    uint64_t nrc = 0, nsc = 0;
    if (hr && hs) {
        nrc = (hr + (uint64_t)a.capR - 1) / a.capR;
        nsc = s_chunks(hs, nrc, split_all);
    }
    const uint64_t mine = nrc * nsc;
    // warp prefix of the item counts, one reservation per warp
    uint64_t inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    const uint64_t wtot = __shfl_sync(0xffffffffu, inc, 31);
    unsigned wb = 0;
    if (lane == 31 && wtot) wb = atomicAdd(&a.ctrl->nitems, (unsigned)wtot);
    wb = __shfl_sync(0xffffffffu, wb, 31);
    uint64_t off = (uint64_t)wb + inc - mine;
    const bool fits = off + mine <= a.item_cap;  // always, with the host's bound; guarded anyway
    if (mine && !fits) atomicCAS(&a.ctrl->error, 0u, (unsigned)TBG_ERR_CAPACITY);
    if (mine && fits) {
        const uint64_t sstep = (hs + nsc - 1) / nsc;
        const uint64_t rb = __ldcg(a.r.base + f), sb = __ldcg(a.s.base + f);
        for (uint64_t rc = 0; rc < nrc; rc++) {
            for (uint64_t sc = 0; sc < nsc; sc++) {
                Item it;
                it.part = (uint32_t)f;
                it.r_off = rb + rc * (uint64_t)a.capR;
                it.r_len = (uint32_t)umin64((uint64_t)a.capR, hr - rc * (uint64_t)a.capR);
                it.s_off = sb + sc * sstep;
                it.s_len = umin64(sstep, hs - sc * sstep);
                a.items[off++] = it;
            }
        }
    }
    const unsigned ne = __popc(__ballot_sync(0xffffffffu, mine != 0));
    if (lane == 0 && ne) atomicAdd(&a.ctrl->nonempty, (unsigned long long)ne);
}


// Takes a ticket of *ctr after this CTA's writes; true for all threads of the
// CTA that takes the last of `n`, which then sees the others' writes, and
// leaves the counter at zero.
__device__ bool last_of(unsigned *ctr, unsigned n, int tid, bool *flag) {
    __syncthreads();  // this CTA's writes come before its ticket
    if (tid == 0) {
        __threadfence();
        const bool last = atomicAdd(ctr, 1u) == n - 1;
        if (last) {
            *ctr = 0;
            __threadfence();
        }
        *flag = last;
    }
    __syncthreads();
    return *flag;
}

// Column scans of relation R in CTAs [0, cols of it), of S in the rest.  With
// t.plan, each relation's last CTA scans its bases; with t.items, the CTA that
// finishes the last relation of the launch plans the work items.
__global__ void __launch_bounds__(PLAN_THREADS) k_colscan(ColScan r, ColScan s, PlanTail t) {
    dep_wait();
    dep_trigger();
    __shared__ uint32_t seg[32][33];
    __shared__ uint64_t scratch[PLAN_THREADS / 32 + 1];
    __shared__ bool flag;
    const int cols_r = (r.P + 31) / 32, cols_s = (s.P + 31) / 32;
    const bool is_s = (int)blockIdx.x >= cols_r;
    const bool totals_only = t.done && t.plan.ctrl->direct;
    if (!is_s) column_scan(r.hist, r.G, r.P, r.totals, blockIdx.x, seg, totals_only);
    else column_scan(s.hist, s.G, s.P, s.totals, blockIdx.x - cols_r, seg, totals_only);
    if (!t.done) return;
    const int tid = threadIdx.y * 32 + threadIdx.x;
    if (!last_of(t.done + is_s, is_s ? cols_s : cols_r, tid, &flag)) return;
    Ctrl *ctrl = t.plan.ctrl;
    const int P = 1 << t.plan.P_log2;
    const RelPlan &rel = is_s ? t.plan.s : t.plan.r;
    plan_bases(rel.hist, rel.base, P, is_s ? &ctrl->max_part_S : &ctrl->max_part_R, tid, scratch);
    if (!t.items) return;
    if (!last_of(t.done + 2, cols_r && cols_s ? 2 : 1, tid, &flag)) return;
    if (tid == 0) ctrl->nitems = 0;
    __threadfence();
    __syncthreads();
    for (int b = 0; b * PLAN_THREADS < P; b++) plan_block(t.plan, b, tid, scratch);
}

__global__ void __launch_bounds__(PLAN_THREADS) k_plan(PlanArgs a) {
    __shared__ uint64_t scratch[PLAN_THREADS / 32 + 1];
    plan_block(a, blockIdx.x, threadIdx.x, scratch);
}

// ---------------------------------------------------------------------------
// K4 pass 1: CTA c scatters chunk c by d1.  With one pass, d1 is f itself.
// Both passes take up to two relations (the second one null for one): S's
// CTAs come first, and R's, fewer and shorter, fill the last wave.
// ---------------------------------------------------------------------------
template <int THREADS, class Out>
__device__ __forceinline__ void part_pass1(const PartArgs &a, const int c) {
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto &sm = *reinterpret_cast<PassSmem<THREADS> *>(smem_raw);
    const int tid = threadIdx.x;
    const int P = 1 << (a.b1 + a.b2);
    const int F = 1 << a.b1;
    const uint32_t *pre = a.pre + (uint64_t)c * P;
    const uint32_t *nxt = c + 1 < a.G ? a.pre + (uint64_t)(c + 1) * P : a.totals;
    // cursors: sum the chunk's prefix over each pass-1 digit's final partitions
    // (delta[0] holds the chunk's row count per pass-1 digit until the scatter)
    uint32_t *rows1 = sm.delta[0];
    for (int i = tid; i < F; i += THREADS) {
        sm.cursor[i] = 0;
        rows1[i] = 0;
    }
    __syncthreads();
    {
        // each thread sums a contiguous run of f (one pass-1 digit per flush)
        const int per = P >= THREADS ? P / THREADS : 1;
        const int f0 = tid * per;
        uint32_t acc_c = 0, acc_t = 0;
        int cur_s = -1;
        for (int f = f0; f < f0 + per && f < P; f++) {
            const int s = f >> a.b2;
            if (s != cur_s) {
                if (cur_s >= 0) {
                    atomicAdd(&sm.cursor[cur_s], acc_c);
                    atomicAdd(&rows1[cur_s], acc_t);
                }
                cur_s = s;
                acc_c = acc_t = 0;
            }
            acc_c += pre[f];
            acc_t += nxt[f] - pre[f];
        }
        if (cur_s >= 0) {
            atomicAdd(&sm.cursor[cur_s], acc_c);
            atomicAdd(&rows1[cur_s], acc_t);
        }
    }
    __syncthreads();
    for (int s = tid; s < F; s += THREADS) {
        const uint32_t cur = (uint32_t)a.base[(uint64_t)s << a.b2] + sm.cursor[s];
        sm.cursor[s] = cur;
        if (a.off1) {
            a.off1[(uint64_t)c * F + s] = cur;
            a.cnt1[(uint64_t)c * F + s] = rows1[s];
        }
    }
    __syncthreads();
    const uint64_t lo = (uint64_t)c * a.chunk;
    const uint64_t hi = a.chunk_len ? lo + a.chunk_len[c] : umin64(a.n, lo + a.chunk);
    part_range<THREADS, Out>(static_cast<const Row *>(a.in), lo, hi, a.n, static_cast<Out *>(a.out), (uint32_t)a.n, a.d1,
                             sm, a.err);
}

// ---------------------------------------------------------------------------
// K5 pass 2: unit (c, s), s-major, scatters by d2 within pass-1 partition s.
// ---------------------------------------------------------------------------
template <int THREADS, class E>
__device__ __forceinline__ void part_pass2(const PartArgs &a, const unsigned unit) {
    if (a.skip && *a.skip) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto &sm = *reinterpret_cast<PassSmem<THREADS, E> *>(smem_raw);
    const int F1 = 1 << a.b1, F2 = 1 << a.b2;
    const int P = F1 * F2;
    const int ngroups = (a.G + a.group - 1) / a.group;
    const int s = (int)(unit / ngroups), g = (int)(unit % ngroups);
    const int c0 = g * a.group, c1 = min(a.G, c0 + a.group) - 1;
    // chunk c's rows of partition s follow chunk c-1's in the pass-1 output,
    // so a group of chunks is one contiguous range with one cursor per digit
    const uint64_t lo = a.off1[(uint64_t)c0 * F1 + s];
    const uint64_t hi = (uint64_t)a.off1[(uint64_t)c1 * F1 + s] + a.cnt1[(uint64_t)c1 * F1 + s];
    if (lo >= hi) return;
    for (int d = threadIdx.x; d < F2; d += THREADS) {
        const uint64_t f = ((uint64_t)s << a.b2) | d;
        sm.cursor[d] = (uint32_t)a.base[f] + a.pre[(uint64_t)c0 * P + f];
    }
    __syncthreads();
    part_range<THREADS, E>(static_cast<const E *>(a.in), lo, hi, a.n, static_cast<E *>(a.out), (uint32_t)a.n, a.d2, sm,
                           a.err);
}

// The two relations of a launch take two copies of the pass in the code:
// reading the arguments through one selected pointer costs registers that the
// pass does not have (64 of 64 in use; with it the passes ran 5% slower).
// E: what the partitions hold, rows or bare keys.
template <int THREADS, class E>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
    k_part_pass1(const __grid_constant__ PartArgs a, const __grid_constant__ PartArgs b) {
    dep_wait();
    dep_trigger();
    if (blockIdx.x < (unsigned)a.G) part_pass1<THREADS, E>(a, blockIdx.x);
    else part_pass1<THREADS, E>(b, blockIdx.x - a.G);
}

template <int THREADS, class E>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
    k_part_pass2(const __grid_constant__ PartArgs a, const __grid_constant__ PartArgs b) {
    dep_wait();
    dep_trigger();
    const unsigned units = (unsigned)((a.G + a.group - 1) / a.group) << a.b1;
    if (blockIdx.x < units) part_pass2<THREADS, E>(a, blockIdx.x);
    else part_pass2<THREADS, E>(b, blockIdx.x - units);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
int hist_ctas_per_sm(int P_log2) {
    const size_t smem = ((size_t)1 << P_log2) * 4;
    int n = 0;
    smem_limit((const void *)k_hist_chunks, smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_hist_chunks, HIST_THREADS, smem);
    return n < 1 ? 1 : n;
}

cudaError_t launch_hist_chunks(const Row *in, uint64_t n, uint64_t chunk, int G, uint32_t *hist,
                               int P_log2, RadixF rf, cudaStream_t st, unsigned long long *oor, uint32_t range_max) {
    const int nbins = 1 << P_log2;
    const size_t smem = (size_t)nbins * 4;
    cudaError_t e = smem_limit((const void *)k_hist_chunks, smem);
    if (e != cudaSuccess) return e;
    e = launch_dep(k_hist_chunks, G, HIST_THREADS, smem, st, in, n, chunk, hist, nbins, rf, oor, range_max);
    count_launch();
    return e;
}

cudaError_t launch_colscan(uint32_t *hist, int G, int P, uint32_t *totals, cudaStream_t st) {
    k_colscan<<<(P + 31) / 32, dim3(32, 32), 0, st>>>(ColScan{hist, totals, G, P}, ColScan{}, PlanTail{});
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_colscan_plan(const ColScan &r, const ColScan &s, const PlanTail &t, cudaStream_t st) {
    const cudaError_t e = launch_dep(k_colscan, (r.P + 31) / 32 + (s.P + 31) / 32, dim3(32, 32), 0, st, r, s, t);
    count_launch();
    return e;
}

cudaError_t launch_plan(const PlanArgs &a, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(&a.ctrl->nitems, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    const int P = 1 << a.P_log2;
    k_plan<<<(P + PLAN_THREADS - 1) / PLAN_THREADS, PLAN_THREADS, 0, st>>>(a);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_part_pass1(const PartArgs &a, const PartArgs *b, cudaStream_t st) {
    constexpr int T = PASS1_THREADS;
    const size_t smem = sizeof(PassSmem<T>);
    auto kern = a.keys ? k_part_pass1<T, uint32_t> : k_part_pass1<T, Row>;
    cudaError_t e = smem_limit((const void *)kern, smem);
    if (e != cudaSuccess) return e;
    e = launch_dep(kern, a.G + (b ? b->G : 0), T, smem, st, a, b ? *b : a);
    count_launch();
    return e;
}

cudaError_t launch_part_pass2(const PartArgs &a, const PartArgs *b, cudaStream_t st) {
    constexpr int T = PASS2_THREADS;
    const size_t smem = a.keys ? sizeof(PassSmem<T, uint32_t>) : sizeof(PassSmem<T>);
    auto kern = a.keys ? k_part_pass2<T, uint32_t> : k_part_pass2<T, Row>;
    cudaError_t e = smem_limit((const void *)kern, smem);
    if (e != cudaSuccess) return e;
    auto units = [](const PartArgs &p) { return (uint64_t)((p.G + p.group - 1) / p.group) << p.b1; };
    e = launch_dep(kern, (unsigned)(units(a) + (b ? units(*b) : 0)), T, smem, st, a, b ? *b : a);
    count_launch();
    return e;
}

}  // namespace tbg
