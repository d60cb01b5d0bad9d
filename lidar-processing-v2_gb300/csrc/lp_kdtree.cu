// lp_kdtree.cu — dynamic-radius outlier removal exactly as the reference's kd-tree search leaves it.
//
// Reference: NoiseRemover::filter (lidar_processing_lib/src/noise_remover.cpp:38-68) over
// KDTree::rebuild (kdtree.hpp:161-214) and KDTree::radius_search_k_nearest (kdtree.hpp:339-397).
// Per point, in input order: squared radius r2 = max(float(s2 * double(x*x + y*y)), rmin^2); a
// depth-first search from the root counts nodes with d0 + (d1 + d2) <= r2 (dk = (q_k - p_k)^2 in
// binary32, query first) and stops at min_neighbours; fewer found means NOISE. The search's stack
// is a member of the tree and is not cleared when the search stops early: the next point's search
// pushes the root on top of what is left, and once its own subtrees are exhausted it carries on
// through the subtrees earlier searches left behind, counting points there again. A point with
// fewer than min_neighbours true neighbours can therefore still reach the count. This file
// reproduces that sequence exactly (every scan starts with an empty stack, as a new NoiseRemover):
//
//   1. Tree (k_kt_level): the reference builds its tree by std::nth_element on the middle of
//      each range (x, y, z by depth); which of several points with equal coordinates lands on
//      which side depends on that library routine's swaps. The build replays libstdc++'s
//      introselect step for step (median of three, unguarded Hoare partition, insertion sort at
//      three elements, heap selection at the depth limit). Large ranges: one CTA per range, the
//      Hoare partition replayed in parallel (the t-th element >= pivot from the left is swapped
//      with the t-th element <= pivot from the right while the first lies left of the second);
//      ranges of at most kKtSmall points finish their whole subtree in shared memory. Node
//      children follow from the range arithmetic alone, so a node record is its point and its
//      subtree size; subtree boxes (k_kt_box_level) serve the skip test of steps 3 and 4.
//   2. Own search (k_kt_own, one thread per point, taken in tree order): the point's search from
//      the root, in the reference's push order, until min_neighbours or exhaustion. A point that reaches the
//      count leaves the rest of its stack behind: those entries go to a pool, then into one
//      array in point order (k_kt_flat). Points that exhaust their own search ("short" points)
//      are listed in order (k_kt_short).
//   3. Own segment (k_kt_segment, one thread per short point): the stack a short point meets is
//      the leftovers of the points since the previous short point (a contiguous piece of the
//      array, newest on top) above whatever the previous short point left. The point walks its
//      piece from the top; an entry whose subtree box is farther than the radius is consumed
//      without a match (skipped); the others are searched exactly. Reaching the count there
//      decides the point (VALID) and records where it stopped and the entries it left.
//   4. Candidates (short points step 3 did not decide). k_kt_spec, one thread per
//      candidate: the walk through the pieces pushed since the previous candidate, as if nothing
//      lay below them, which is exact whenever the previous candidate emptied the stack (running
//      out of entries is NOISE). k_kt_spec_next, one thread per candidate whose walk ran out right
//      after one whose walk stopped: the walk on through the pieces that stop leaves, which lie
//      on top of whatever was below. k_kt_run, one CTA per stopped candidate: it and the candidates
//      after it up to the next that stopped, as if nothing lay below its pieces: each continues into
//      them, the threads searching 256 entries at a time, an ordered prefix of their counts finding
//      the stop, until one empties them. k_kt_chain, one CTA per scan: the runs in order, with what
//      earlier runs left; only where that is not empty and a run emptied its own pieces do candidates
//      search on (about one run in twenty).
// The result equals the reference's sequential search bit for bit (same binary32 expressions,
// same visiting order, same stop points); the tree's node positions equal the reference's.
#include <cooperative_groups.h>

#include "lp_batch.cuh"
#include "lp_common.cuh"
#include "lp_stages.hpp"

namespace cg = cooperative_groups;

namespace lpg
{
namespace
{
constexpr uint32_t kKtSmall = 2048;    // ranges built in shared memory by one CTA
constexpr uint32_t kKtHuge = 65536;    // ranges partitioned by a cluster of kKtCluster CTAs
constexpr uint32_t kKtFew = 6144;      // the same on levels of few ranges
constexpr uint32_t kKtStage = 4096;   // ranges finished in shared memory by one CTA
constexpr uint32_t kKtBlockMin = 512; // where a round by the whole CTA still beats one by a warp
constexpr uint32_t kKtClusterMin = kKtStage; // the cluster's rounds run while the range exceeds this
constexpr int kKtSmallThreads = 512; // at most
constexpr int kKtCluster = 8;
constexpr uint32_t kKtWarpMin = 16;    // ranges of at most this many points finish on one thread
constexpr int kKtThreads = 512;        // tree build CTAs
constexpr int kKtStack = 64;           // search stack entries (>= tree depth + 1 for 2^62 points)
constexpr uint32_t kNone = 0xffffffffu;

// Stack entries: node position (scan-local) << 2 | axis.
__device__ __forceinline__ uint32_t kt_entry(uint32_t m, int ax)
{
    return (m << 2) | static_cast<uint32_t>(ax);
}

__device__ __forceinline__ float kt_coord(const float4& r, int ax)
{
    return ax == 0 ? r.x : (ax == 1 ? r.y : r.z);
}

__device__ __forceinline__ float kt_radius2(const ScanDev& sd, const float4& p)
{
    // noise_remover.cpp:55-57: float products and sum, widened, scaled, narrowed, floored
    const double rho2 = static_cast<double>((p.x * p.x) + (p.y * p.y));
    return fmaxf(__double2float_rn(sd.dror_s2 * rho2), sd.dror_rmin2);
}

__device__ __forceinline__ uint32_t floor_log2_u(uint32_t v)
{
    return 31u - static_cast<uint32_t>(__clz(v));
}

// Range of node slot j (0 <= j < 2^level) of the implicit tree over [0, n): the bits of j from the
// top choose left (0) or right (1) at each level. Returns false where the range does not exist.
// *plen receives the parent's length (n for the root).
__device__ __forceinline__ bool kt_range(uint32_t n, int level, uint32_t j, uint32_t& b, uint32_t& e, uint32_t* plen)
{
    b = 0;
    e = n;
    uint32_t parent = n;
    for (int l = level - 1; l >= 0; --l)
    {
        if (e <= b)
            return false;
        const uint32_t mid = b + (e - b) / 2;
        parent = e - b;
        if ((j >> l) & 1u)
            b = mid + 1;
        else
            e = mid;
    }
    if (plen)
        *plen = parent;
    return e > b;
}

// ---------------------------------------------------------------------------------------------
// libstdc++ introselect, one thread (std::nth_element as GCC's <bits/stl_algo.h> performs it).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void kt_swap(float4* a, uint32_t i, uint32_t j)
{
    const float4 t = a[i];
    a[i] = a[j];
    a[j] = t;
}

// The median of a[first + 1], a[mid], a[last - 1] is swapped into a[first].
__device__ void kt_median_to_first(float4* a, uint32_t first, uint32_t last, int ax)
{
    const uint32_t x = first + 1, y = first + (last - first) / 2, z = last - 1;
    const float vx = kt_coord(a[x], ax), vy = kt_coord(a[y], ax), vz = kt_coord(a[z], ax);
    uint32_t m;
    if (vx < vy)
        m = (vy < vz) ? y : ((vx < vz) ? z : x);
    else
        m = (vx < vz) ? x : ((vy < vz) ? z : y);
    kt_swap(a, first, m);
}

// Unguarded Hoare partition of [first + 1, last) around a[first]; returns the cut. The median of
// three guarantees an element >= pivot and one <= pivot inside the range, which stop the scans;
// the explicit bounds only keep a malformed input (NaN coordinates) inside the range.
__device__ uint32_t kt_partition_seq(float4* a, uint32_t first, uint32_t last, int ax)
{
    const float p = kt_coord(a[first], ax);
    uint32_t lo = first + 1, hi = last;
    for (;;)
    {
        while (lo + 1 < last && kt_coord(a[lo], ax) < p)
            ++lo;
        --hi;
        while (hi > first && p < kt_coord(a[hi], ax))
            --hi;
        if (!(lo < hi))
            return lo;
        kt_swap(a, lo, hi);
        ++lo;
    }
}

__device__ void kt_insertion(float4* a, uint32_t first, uint32_t last, int ax)
{
    if (first == last)
        return;
    for (uint32_t i = first + 1; i < last; ++i)
    {
        const float4 v = a[i];
        const float kv = kt_coord(v, ax);
        if (kv < kt_coord(a[first], ax))
        {
            for (uint32_t j = i; j > first; --j)
                a[j] = a[j - 1];
            a[first] = v;
        }
        else
        {
            uint32_t j = i;
            while (j > first + 1 && kv < kt_coord(a[j - 1], ax))
            {
                a[j] = a[j - 1];
                --j;
            }
            a[j] = v;
        }
    }
}

// Max-heap sift of value v from `hole` in a[base, base + len) (std::__adjust_heap + __push_heap).
__device__ void kt_sift(float4* a, uint32_t base, uint32_t hole, uint32_t len, float4 v, int ax)
{
    const uint32_t top = hole;
    uint32_t child = hole;
    while (len >= 2 && child < (len - 1) / 2)
    {
        child = 2 * (child + 1);
        if (kt_coord(a[base + child], ax) < kt_coord(a[base + child - 1], ax))
            --child;
        a[base + hole] = a[base + child];
        hole = child;
    }
    if ((len & 1u) == 0 && len >= 2 && child == (len - 2) / 2)
    {
        child = 2 * (child + 1);
        a[base + hole] = a[base + child - 1];
        hole = child - 1;
    }
    const float kv = kt_coord(v, ax);
    uint32_t parent = (hole - 1) / 2;
    while (hole > top && kt_coord(a[base + parent], ax) < kv)
    {
        a[base + hole] = a[base + parent];
        hole = parent;
        parent = (hole - 1) / 2;
    }
    a[base + hole] = v;
}

// std::__heap_select(first, middle, last) then the swap of first and nth (introselect at the depth
// limit): a max-heap of [first, nth], every later element smaller than its top replaces it.
__device__ void kt_heap_select(float4* a, uint32_t first, uint32_t nth, uint32_t last, int ax)
{
    const uint32_t mid = nth - first + 1;
    if (mid >= 2)
        for (uint32_t parent = (mid - 2) / 2;; --parent)
        {
            kt_sift(a, first, parent, mid, a[first + parent], ax);
            if (parent == 0)
                break;
        }
    for (uint32_t i = first + mid; i < last; ++i)
        if (kt_coord(a[i], ax) < kt_coord(a[first], ax))
        {
            const float4 v = a[i];
            a[i] = a[first];
            kt_sift(a, first, 0, mid, v, ax);
        }
    kt_swap(a, first, nth);
}

// Continues an introselect of nth in [first, last) with `depth` rounds left, on one thread.
__device__ void kt_select_seq(float4* a, uint32_t first, uint32_t nth, uint32_t last, int depth, int ax)
{
    while (last - first > 3)
    {
        if (depth == 0)
        {
            kt_heap_select(a, first, nth, last, ax);
            return;
        }
        --depth;
        kt_median_to_first(a, first, last, ax);
        const uint32_t cut = kt_partition_seq(a, first, last, ax);
        if (cut <= nth)
            first = cut;
        else
            last = cut;
    }
    kt_insertion(a, first, last, ax);
}

// ---------------------------------------------------------------------------------------------
// One partition round by a whole CTA: median of three into a[first], then the unguarded Hoare
// partition of [first + 1, last) replayed in parallel. With L_t the t-th position (from the
// left) holding a value >= pivot and R_t the t-th (from the right) holding a value <= pivot, the
// sequential loop swaps L_t with R_t for every t with L_t < R_t (T such pairs; these pairs are
// disjoint) and then stops at min(L_{T+1}, R_T) (L_1 when T = 0): the left scan meets either the
// next original candidate or the element it swapped to R_T. ge/le receive the candidate
// positions in ascending order (le reversed gives R). Returns the cut.
// ---------------------------------------------------------------------------------------------
// T and the cut from the candidate lists, by a whole warp: the predicate ge[t - 1] < le[nle - t] holds
// for t up to T, found with 32 probes a step (three or four dependent loads instead of sixteen).
template <typename I>
__device__ __forceinline__ void kt_find_cut(const I* ge, uint32_t nge, const I* le, uint32_t nle, uint32_t& T, uint32_t& cut)
{
    const uint32_t lane = lane_id();
    uint32_t lo = 0, hi = min(nge, nle);
    while (lo < hi)
    {
        const uint32_t w = (hi - lo + 31u) / 32u;
        const uint32_t t = min(lo + (lane + 1u) * w, hi);
        const uint32_t k = static_cast<uint32_t>(__popc(__ballot_sync(0xffffffffu, ge[t - 1u] < le[nle - t])));
        const uint32_t above = min(lo + (k + 1u) * w, hi); // the first probe that failed (none: k = 32)
        lo = min(lo + k * w, hi);
        hi = (k == 32u) ? hi : above - 1u;
        if (k == 32u)
            lo = hi;
    }
    T = lo;
    cut = (T == 0u) ? static_cast<uint32_t>(ge[0])
                    : min(T < nge ? static_cast<uint32_t>(ge[T]) : 0xffffffffu, static_cast<uint32_t>(le[nle - T]));
}

// A warp's part of a partition round: elements [c0, c1) after `lo`, in rows of 32 (lane = element, so
// loads and list writes are contiguous), kKtRows rows in flight. Counts first; with the counts of the
// warps before it known, the second pass writes the positions without any barrier in between.
constexpr int kKtRows = 8;

__device__ __forceinline__ void kt_count_rows(const float4* a, uint32_t lo, uint32_t c0, uint32_t c1, int ax, float p,
                                              uint32_t& nge, uint32_t& nle)
{
    const float* key = reinterpret_cast<const float*>(a + lo) + ax;
    uint32_t g = 0, l = 0;
    for (uint32_t base = c0; base < c1; base += 32u * kKtRows)
    {
        float v[kKtRows];
#pragma unroll
        for (int u = 0; u < kKtRows; ++u)
        {
            const uint32_t k = base + static_cast<uint32_t>(u) * 32u + lane_id();
            v[u] = (k < c1) ? key[4ull * k] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < kKtRows; ++u)
        {
            const bool in = base + static_cast<uint32_t>(u) * 32u + lane_id() < c1;
            g += (in && !(v[u] < p)) ? 1u : 0u;
            l += (in && !(p < v[u])) ? 1u : 0u;
        }
    }
    nge = warp_sum(g);
    nle = warp_sum(l);
}

template <typename I>
__device__ __forceinline__ void kt_write_rows(const float4* a, uint32_t lo, uint32_t c0, uint32_t c1, int ax, float p, I* ge,
                                              uint32_t og, I* le, uint32_t ol)
{
    const float* key = reinterpret_cast<const float*>(a + lo) + ax;
    const uint32_t below = (1u << lane_id()) - 1u;
    for (uint32_t base = c0; base < c1; base += 32u * kKtRows)
    {
        float v[kKtRows];
#pragma unroll
        for (int u = 0; u < kKtRows; ++u)
        {
            const uint32_t k = base + static_cast<uint32_t>(u) * 32u + lane_id();
            v[u] = (k < c1) ? key[4ull * k] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < kKtRows; ++u)
        {
            const uint32_t k = base + static_cast<uint32_t>(u) * 32u + lane_id();
            const bool g = k < c1 && !(v[u] < p), l = k < c1 && !(p < v[u]);
            const uint32_t bg = __ballot_sync(0xffffffffu, g), bl = __ballot_sync(0xffffffffu, l);
            if (g)
                ge[og + static_cast<uint32_t>(__popc(bg & below))] = static_cast<I>(lo + k);
            if (l)
                le[ol + static_cast<uint32_t>(__popc(bl & below))] = static_cast<I>(lo + k);
            og += static_cast<uint32_t>(__popc(bg));
            ol += static_cast<uint32_t>(__popc(bl));
        }
    }
}

// The swaps t, t + step, ... below T, four pairs in flight (the pairs are disjoint).
template <typename I>
__device__ __forceinline__ void kt_swap_pairs(float4* a, const I* ge, const I* le, uint32_t nle, uint32_t T, uint32_t t0,
                                              uint32_t step)
{
    for (uint32_t t = t0; t < T; t += 4u * step)
    {
        uint32_t x[4], y[4];
        float4 vx[4], vy[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
        {
            const uint32_t q = min(t + u * step, T - 1u);
            x[u] = ge[q];
            y[u] = le[nle - 1u - q];
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
        {
            vx[u] = a[x[u]];
            vy[u] = a[y[u]];
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
            if (t + u * step < T)
            {
                a[x[u]] = vy[u];
                a[y[u]] = vx[u];
            }
    }
}

struct KtShared
{
    uint2 warp_cnt[32];
    uint32_t bcast[2];
};

template <typename I>
__device__ __forceinline__ uint32_t kt_round_block(float4* a, uint32_t first, uint32_t last, int ax, I* ge, I* le, KtShared& sh)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t nwarps = blockDim.x >> 5;
    if (tid == 0)
        kt_median_to_first(a, first, last, ax);
    __syncthreads();
    const float p = kt_coord(a[first], ax);
    const uint32_t lo = first + 1, n = last - lo;
    const uint32_t part = ((n + nwarps - 1u) / nwarps + 31u) & ~31u;
    const uint32_t c0 = min(n, warp * part), c1 = min(n, c0 + part);
    uint32_t cge, cle;
    kt_count_rows(a, lo, c0, c1, ax, p, cge, cle);
    if (lane == 0)
        sh.warp_cnt[warp] = make_uint2(cge, cle);
    __syncthreads();
    const uint2 wc = (lane < nwarps) ? sh.warp_cnt[lane] : make_uint2(0u, 0u);
    const uint32_t ig = warp_incl_scan(wc.x), il = warp_incl_scan(wc.y);
    const uint32_t nge = __shfl_sync(0xffffffffu, ig, 31), nle = __shfl_sync(0xffffffffu, il, 31);
    kt_write_rows(a, lo, c0, c1, ax, p, ge, __shfl_sync(0xffffffffu, ig - wc.x, static_cast<int>(warp)), le,
                  __shfl_sync(0xffffffffu, il - wc.y, static_cast<int>(warp)));
    __syncthreads();
    if (warp == 0)
    {
        uint32_t T, cut;
        kt_find_cut(ge, nge, le, nle, T, cut);
        if (lane == 0)
        {
            sh.bcast[0] = T;
            sh.bcast[1] = cut;
        }
    }
    __syncthreads();
    const uint32_t T = sh.bcast[0], cut = sh.bcast[1];
    kt_swap_pairs(a, ge, le, nle, T, tid, blockDim.x);
    __syncthreads();
    return cut;
}

__device__ void kt_select_warp(float4* a, uint32_t first, uint32_t nth, uint32_t last, int ax, uint16_t* ge,
                               uint16_t* le, int depth);

// Continues an introselect of nth in [first, last) of a (shared memory, at most kKtStage points; lists
// of uint16) by a whole CTA: block rounds while the range is worth them, then warp 0.
__device__ __forceinline__ void kt_select_staged(float4* a, uint32_t first, uint32_t nth, uint32_t last, int depth, int ax,
                                                 uint16_t* ge, uint16_t* le, KtShared& sh)
{
    while (last - first > kKtBlockMin && depth > 0)
    {
        --depth;
        const uint32_t cut = kt_round_block(a, first, last, ax, ge, le, sh);
        if (cut <= nth)
            first = cut;
        else
            last = cut;
    }
    if (threadIdx.x < 32)
        kt_select_warp(a, first, nth, last, ax, ge, le, depth);
    __syncthreads();
}

// Continues an introselect of nth in [first, last) (global memory) with `depth` rounds left on a
// whole CTA: parallel rounds while the range exceeds kKtStage points, then the range is copied to
// shared memory (srec, with 2 kKtStage list entries at slist) and finished there. The depth-limit
// fallback on a larger range runs on thread 0.
__device__ void kt_select_block(float4* a, uint32_t first, uint32_t nth, uint32_t last, int depth, int ax,
                                uint32_t* ge, uint32_t* le, KtShared& sh, float4* srec, uint16_t* slist)
{
    while (last - first > kKtStage && depth > 0)
    {
        --depth;
        const uint32_t cut = kt_round_block(a, first, last, ax, ge, le, sh);
        if (cut <= nth)
            first = cut;
        else
            last = cut;
    }
    const uint32_t len = last - first;
    if (len > kKtStage)
    {
        if (threadIdx.x == 0)
            kt_select_seq(a, first, nth, last, depth, ax);
        __syncthreads();
        return;
    }
    for (uint32_t k = threadIdx.x; k < len; k += blockDim.x)
        srec[k] = a[first + k];
    __syncthreads();
    kt_select_staged(srec, 0, nth - first, len, depth, ax, slist, slist + len, sh);
    for (uint32_t k = threadIdx.x; k < len; k += blockDim.x)
        a[first + k] = srec[k];
    __syncthreads();
}

// One partition round by one warp on a[first, last) in shared memory (the parallel Hoare replay of
// kt_round_block, 32 elements per step with ballots); ge/le hold the candidate positions.
__device__ uint32_t kt_round_warp(float4* a, uint32_t first, uint32_t last, int ax, uint16_t* ge, uint16_t* le)
{
    const uint32_t lane = lane_id();
    if (lane == 0)
        kt_median_to_first(a, first, last, ax);
    __syncwarp();
    const float p = kt_coord(a[first], ax);
    const uint32_t lo = first + 1, n = last - lo;
    const uint32_t below = (1u << lane) - 1u;
    uint32_t nge = 0, nle = 0;
    for (uint32_t base = 0; base < n; base += 32)
    {
        const uint32_t idx = base + lane;
        bool g = false, l = false;
        if (idx < n)
        {
            const float v = kt_coord(a[lo + idx], ax);
            g = !(v < p);
            l = !(p < v);
        }
        const uint32_t bg = __ballot_sync(0xffffffffu, g), bl = __ballot_sync(0xffffffffu, l);
        if (g)
            ge[nge + __popc(bg & below)] = static_cast<uint16_t>(lo + idx);
        if (l)
            le[nle + __popc(bl & below)] = static_cast<uint16_t>(lo + idx);
        nge += __popc(bg);
        nle += __popc(bl);
    }
    __syncwarp();
    uint32_t T, cut;
    kt_find_cut(ge, nge, le, nle, T, cut);
    for (uint32_t t = lane; t < T; t += 32)
        kt_swap(a, ge[t], le[nle - 1 - t]);
    __syncwarp();
    return cut;
}

// Continues an introselect of nth in [first, last) (shared memory) with `depth` rounds left on one
// warp: parallel rounds while the range holds more than kKtWarpMin points, then lane 0 as written.
// (A parallel round replays the sequential partition exactly at any size; a small range on one
// thread is a chain of dependent shared-memory accesses, and ranges on neighbouring threads diverge.)
__device__ void kt_select_warp(float4* a, uint32_t first, uint32_t nth, uint32_t last, int ax, uint16_t* ge,
                               uint16_t* le, int depth)
{
    while (last - first > kKtWarpMin && depth > 0)
    {
        --depth;
        const uint32_t cut = kt_round_warp(a, first, last, ax, ge, le);
        if (cut <= nth)
            first = cut;
        else
            last = cut;
    }
    if (lane_id() == 0)
        kt_select_seq(a, first, nth, last, depth, ax);
    __syncwarp();
}

// Subtree of [b0, e0) (at depth d0 of the tree, at most kKtSmall points) built in shared memory;
// node records get their subtree size in .w (the input index it carried goes to idx); subtree
// boxes are written bottom-up.
__device__ void kt_build_small(float4* g, float4* box, uint32_t* idx, uint32_t b0, uint32_t e0, int d0, float4* s,
                               uint16_t* lists, KtShared& sh)
{
    const uint32_t n = e0 - b0;
    const uint32_t warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x)
        s[k] = g[b0 + k];
    __syncthreads();
    // the longest range at depth d has floor(n / 2^d) points (a range of L splits into floor(L/2)
    // and ceil(L/2) - 1), so depths 0 .. floor(log2 n) hold ranges. Ranges above kKtWarpMin: one warp
    // each (positions of range [b, e) in lists[2b, 2e)); the rest: one thread each.
    const int maxd = static_cast<int>(floor_log2_u(n));
    for (int d = 0; d <= maxd; ++d)
    {
        const uint32_t slots = 1u << d;
        if (d == 0 && n > kKtBlockMin)
            kt_select_staged(s, 0, n / 2, n, 2 * static_cast<int>(floor_log2_u(n)), d0 % 3, lists, lists + n, sh);
        else if ((n >> d) > kKtWarpMin)
            for (uint32_t j = warp; j < slots; j += nwarps)
            {
                uint32_t b, e;
                if (kt_range(n, d, j, b, e, nullptr) && e - b > kKtWarpMin)
                    kt_select_warp(s, b, b + (e - b) / 2, e, (d0 + d) % 3, lists + 2 * b, lists + 2 * b + (e - b),
                                   2 * static_cast<int>(floor_log2_u(e - b)));
            }
        for (uint32_t j = threadIdx.x; j < slots; j += blockDim.x)
        {
            uint32_t b, e;
            if (kt_range(n, d, j, b, e, nullptr) && e - b <= kKtWarpMin && e - b > 1)
                kt_select_seq(s, b, b + (e - b) / 2, e, 2 * static_cast<int>(floor_log2_u(e - b)), (d0 + d) % 3);
        }
        __syncthreads();
    }
    // subtree sizes and boxes, deepest level first
    for (int d = maxd; d >= 0; --d)
    {
        const uint32_t slots = 1u << d;
        for (uint32_t j = threadIdx.x; j < slots; j += blockDim.x)
        {
            uint32_t b, e;
            if (!kt_range(n, d, j, b, e, nullptr))
                continue;
            const uint32_t m = b + (e - b) / 2;
            float4 p = s[m];
            idx[b0 + m] = __float_as_uint(p.w);
            p.w = __uint_as_float(e - b);
            s[m] = p;
            float4 lo = make_float4(p.x, p.y, p.z, 0.0f), hi = lo;
            if (m > b)
            {
                const uint32_t c = b0 + b + (m - b) / 2;
                const float4 cl = box[2 * c], ch = box[2 * c + 1];
                lo = make_float4(fminf(lo.x, cl.x), fminf(lo.y, cl.y), fminf(lo.z, cl.z), 0.0f);
                hi = make_float4(fmaxf(hi.x, ch.x), fmaxf(hi.y, ch.y), fmaxf(hi.z, ch.z), 0.0f);
            }
            if (m + 1 < e)
            {
                const uint32_t c = b0 + m + 1 + (e - m - 1) / 2;
                const float4 cl = box[2 * c], ch = box[2 * c + 1];
                lo = make_float4(fminf(lo.x, cl.x), fminf(lo.y, cl.y), fminf(lo.z, cl.z), 0.0f);
                hi = make_float4(fmaxf(hi.x, ch.x), fmaxf(hi.y, ch.y), fmaxf(hi.z, ch.z), 0.0f);
            }
            box[2 * (b0 + m)] = lo;
            box[2 * (b0 + m) + 1] = hi;
        }
        __syncthreads();
    }
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x)
        g[b0 + k] = s[k];
}

// One partition round by a cluster of kKtCluster CTAs on a[first, last) (the median of three into
// a[first] by rank 0, then the same parallel Hoare replay as kt_round_block): every CTA takes a
// slice of [first + 1, last), counts its candidates, learns the counts of the slices before it
// through distributed shared memory and writes its positions in order; rank 0 finds T and the cut;
// the swaps are spread over the whole cluster. Cluster barriers order the global-memory steps.
struct KtClusterShared
{
    uint2 warp_cnt[kKtThreads / 32];
    uint32_t cnt[2]; // this CTA's ge, le counts
    uint32_t res[2]; // rank 0: T, cut
};

__device__ uint32_t kt_round_cluster(float4* a, uint32_t first, uint32_t last, int ax, uint32_t* ge, uint32_t* le,
                                     KtClusterShared& sh, cg::cluster_group& cluster)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const uint32_t rank = cluster.block_rank();
    if (rank == 0 && tid == 0)
        kt_median_to_first(a, first, last, ax);
    cluster.sync();
    const float p = kt_coord(a[first], ax);
    const uint32_t lo = first + 1, n = last - lo;
    // warp w of the cluster's nwarps * kKtCluster takes the w-th part of the range
    const uint32_t part = ((n + nwarps * kKtCluster - 1u) / (nwarps * kKtCluster) + 31u) & ~31u;
    const uint32_t c0 = min(n, (rank * nwarps + warp) * part), c1 = min(n, c0 + part);
    uint32_t cge, cle;
    kt_count_rows(a, lo, c0, c1, ax, p, cge, cle);
    if (lane == 0)
        sh.warp_cnt[warp] = make_uint2(cge, cle);
    __syncthreads();
    const uint2 wc = (lane < nwarps) ? sh.warp_cnt[lane] : make_uint2(0u, 0u);
    const uint32_t ig = warp_incl_scan(wc.x), il = warp_incl_scan(wc.y);
    if (tid == 31)
    {
        sh.cnt[0] = ig;
        sh.cnt[1] = il;
    }
    cluster.sync();
    uint32_t og = __shfl_sync(0xffffffffu, ig - wc.x, static_cast<int>(warp));
    uint32_t ol = __shfl_sync(0xffffffffu, il - wc.y, static_cast<int>(warp));
    uint32_t nge = 0, nle = 0;
    for (uint32_t r = 0; r < static_cast<uint32_t>(kKtCluster); ++r)
    {
        const uint32_t* rc = cluster.map_shared_rank(&sh.cnt[0], r);
        const uint32_t g0 = rc[0], l0 = rc[1];
        if (r < rank)
        {
            og += g0;
            ol += l0;
        }
        nge += g0;
        nle += l0;
    }
    kt_write_rows(a, lo, c0, c1, ax, p, ge, og, le, ol);
    cluster.sync();
    if (rank == 0 && warp == 0)
    {
        uint32_t T, cut;
        kt_find_cut(ge, nge, le, nle, T, cut);
        if (lane == 0)
        {
            sh.res[0] = T;
            sh.res[1] = cut;
        }
    }
    cluster.sync();
    const uint32_t* r0 = cluster.map_shared_rank(&sh.res[0], 0);
    const uint32_t T = r0[0], cut = r0[1];
    kt_swap_pairs(a, ge, le, nle, T, rank * blockDim.x + tid, blockDim.x * kKtCluster);
    cluster.sync();
    return cut;
}

// Levels whose ranges exceed kKtHuge: a cluster per range runs the introselect rounds while the
// range is above kKtClusterMin, then its rank 0 finishes it as a single CTA would (a round on one
// CTA reads the range at one SM's share of the bandwidth).
__global__ void __cluster_dims__(kKtCluster, 1, 1) __launch_bounds__(kKtThreads)
    k_kt_level_huge(BatchDev b, int level, uint32_t slots, uint32_t huge)
{
    pdl_enter();
    extern __shared__ float4 kt_smem[];
    __shared__ KtClusterShared csh;
    __shared__ KtShared sh;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t range = blockIdx.x / kKtCluster;
    const uint32_t s = range / slots, j = range % slots;
    if (s >= static_cast<uint32_t>(b.nscan))
        return; // uniform over the cluster
    const ScanDev& sd = b.scans[s];
    uint32_t lb, le;
    if (!kt_range(sd.n_src, level, j, lb, le, nullptr) || le - lb <= huge)
        return; // uniform over the cluster
    float4* g = b.kt + sd.src_off;
    uint32_t* ge = b.kscr + 2ull * sd.src_off + 2ull * lb;
    uint32_t* lq = ge + (le - lb);
    const uint32_t len = le - lb, nth = lb + len / 2;
    uint32_t first = lb, last = le;
    int depth = 2 * static_cast<int>(floor_log2_u(len));
    while (last - first > kKtClusterMin && depth > 0)
    {
        --depth;
        const uint32_t cut = kt_round_cluster(g, first, last, level % 3, ge, lq, csh, cluster);
        if (cut <= nth)
            first = cut;
        else
            last = cut;
    }
    if (cluster.block_rank() == 0)
    {
        // the rest of the introselect on one CTA
        kt_select_block(g, first, nth, last, depth, level % 3, ge, lq, sh, kt_smem,
                        reinterpret_cast<uint16_t*>(kt_smem + kKtStage));
        if (threadIdx.x == 0)
        {
            float4 p = g[nth];
            b.kq[sd.src_off + nth] = __float_as_uint(p.w);
            p.w = __uint_as_float(len);
            g[nth] = p;
        }
    }
    cluster.sync(); // no CTA leaves while another may read its shared memory
}

__global__ void k_kt_load(BatchDev b)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0)
    {
        b.klo_n[b.nsrc] = 0; // the scanned arrays' last slots (totals after the scans)
        b.kshort[b.nsrc] = 0;
        b.kctr[0] = 0;
    }
    if (i >= b.nsrc)
        return;
    const float4 p = b.src[i];
    // the point's input index rides in .w while the build moves the records (saved in kq when the
    // record becomes a node and .w takes its subtree size)
    b.kt[i] = make_float4(p.x, p.y, p.z, __uint_as_float(i));
}

// One level of the build: CTA (scan, slot j). Ranges above kKtSmall (and up to `huge`) are put in order
// around their middle here.
__global__ void __launch_bounds__(kKtThreads) k_kt_level(BatchDev b, int level, uint32_t slots, uint32_t huge)
{
    pdl_enter();
    extern __shared__ float4 kt_smem[];
    __shared__ KtShared sh;
    const uint32_t s = blockIdx.x / slots, j = blockIdx.x % slots;
    if (s >= static_cast<uint32_t>(b.nscan))
        return;
    const ScanDev& sd = b.scans[s];
    uint32_t lb, le;
    if (!kt_range(sd.n_src, level, j, lb, le, nullptr))
        return;
    const uint32_t len = le - lb;
    if (len > huge || len <= kKtSmall)
        return; // k_kt_level_huge, k_kt_small
    float4* g = b.kt + sd.src_off;
    uint32_t* ge = b.kscr + 2ull * sd.src_off + 2ull * lb;
    uint32_t* lq = ge + len;
    const uint32_t nth = lb + len / 2;
    kt_select_block(g, lb, nth, le, 2 * static_cast<int>(floor_log2_u(len)), level % 3, ge, lq, sh, kt_smem,
                    reinterpret_cast<uint16_t*>(kt_smem + kKtStage));
    if (threadIdx.x == 0)
    {
        float4 p = g[nth];
        b.kq[sd.src_off + nth] = __float_as_uint(p.w);
        p.w = __uint_as_float(len);
        g[nth] = p;
    }
}

// A range of at most kKtSmall points whose parent was larger (or the root): its whole subtree in shared
// memory.
__global__ void __launch_bounds__(kKtSmallThreads) k_kt_small(BatchDev b, int level, uint32_t slots)
{
    pdl_enter();
    extern __shared__ float4 kt_smem[];
    __shared__ KtShared sh;
    const uint32_t s = blockIdx.x / slots, j = blockIdx.x % slots;
    if (s >= static_cast<uint32_t>(b.nscan))
        return;
    const ScanDev& sd = b.scans[s];
    uint32_t lb, le, plen;
    if (!kt_range(sd.n_src, level, j, lb, le, &plen) || le - lb > kKtSmall || !(level == 0 || plen > kKtSmall))
        return;
    kt_build_small(b.kt + sd.src_off, b.kbb + 2ull * sd.src_off, b.kq + sd.src_off, lb, le, level, kt_smem,
                   reinterpret_cast<uint16_t*>(kt_smem + kKtSmall), sh);
}

// Boxes of the nodes above the shared-memory subtrees, one level at a time from the bottom.
__global__ void k_kt_box_level(BatchDev b, int level, uint32_t slots)
{
    pdl_enter();
    const uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint32_t s = static_cast<uint32_t>(t / slots), j = static_cast<uint32_t>(t % slots);
    if (s >= static_cast<uint32_t>(b.nscan))
        return;
    const ScanDev& sd = b.scans[s];
    uint32_t lb, le;
    if (!kt_range(sd.n_src, level, j, lb, le, nullptr) || le - lb <= kKtSmall)
        return;
    const float4* g = b.kt + sd.src_off;
    float4* box = b.kbb + 2ull * sd.src_off;
    const uint32_t m = lb + (le - lb) / 2;
    const float4 p = g[m];
    float4 lo = make_float4(p.x, p.y, p.z, 0.0f), hi = lo;
    const uint32_t cs[2] = {lb + (m - lb) / 2, m + 1 + (le - m - 1) / 2};
    const bool has[2] = {m > lb, m + 1 < le};
    for (int k = 0; k < 2; ++k)
        if (has[k])
        {
            const float4 cl = box[2 * cs[k]], ch = box[2 * cs[k] + 1];
            lo = make_float4(fminf(lo.x, cl.x), fminf(lo.y, cl.y), fminf(lo.z, cl.z), 0.0f);
            hi = make_float4(fmaxf(hi.x, ch.x), fmaxf(hi.y, ch.y), fmaxf(hi.z, ch.z), 0.0f);
        }
    box[2 * m] = lo;
    box[2 * m + 1] = hi;
}

// ---------------------------------------------------------------------------------------------
// The reference's search (kdtree.hpp:355-388) from the entries on stk[0, sp): pop, count the node
// when within r2 (stopping at k), push both children when the splitting plane is within the
// radius (right first, so the left is searched first) or else the side of the query. Empty
// children are not pushed: the reference pushes and pops them without effect. Returns the count;
// after an early stop stk[0, sp) holds the entries left behind.
// ---------------------------------------------------------------------------------------------
__device__ uint32_t kt_search(const float4* __restrict__ g, uint32_t n, float qx, float qy, float qz, float r2,
                              uint32_t k, uint32_t found, uint32_t* stk, int& sp, bool& overflow)
{
    while (sp > 0)
    {
        const uint32_t e = stk[--sp];
        const uint32_t m = e >> 2;
        const int ax = static_cast<int>(e & 3u);
        if (m >= n || ax > 2)
        {
            overflow = true; // not a node of this tree: reported, never followed
            return found;
        }
        const float4 nd = g[m];
        const float d0 = (qx - nd.x) * (qx - nd.x);
        const float d1 = (qy - nd.y) * (qy - nd.y);
        const float d2 = (qz - nd.z) * (qz - nd.z);
        if (d0 + (d1 + d2) <= r2)
        {
            if (++found >= k)
                return found;
        }
        const uint32_t len = __float_as_uint(nd.w);
        if (len == 0 || m < len / 2 || m - len / 2 + len > n)
        {
            overflow = true; // a subtree size the build did not leave: reported, never followed
            return found;
        }
        const uint32_t lb = m - len / 2;
        const uint32_t llen = m - lb, rlen = len - llen - 1;
        const int nx = (ax == 2) ? 0 : ax + 1;
        const float q = (ax == 0) ? qx : ((ax == 1) ? qy : qz);
        const float delta = kt_coord(nd, ax) - q;
        const bool push_r = (delta * delta <= r2) ? true : !(delta > 0);
        const bool push_l = (delta * delta <= r2) ? true : (delta > 0);
        if (sp + 2 > kKtStack)
        {
            overflow = true;
            return found;
        }
        if (push_r && rlen)
            stk[sp++] = kt_entry(m + 1 + rlen / 2, nx);
        if (push_l && llen)
            stk[sp++] = kt_entry(lb + llen / 2, nx);
    }
    return found;
}

// A subtree whose box lies farther than the radius holds no match: the reference's search
// through it ends without counting anything. The box distance is formed in binary32 exactly as
// kt_search forms a point's distance (per-axis difference, square, d0 + (d1 + d2)). Rounding to
// nearest is monotone and odd, so for every point p of the box |fl(q - p)| >= fl(gap) on each axis
// (the gap being the box's bound minus q, or 0 inside the slab), and each square and partial sum of
// p's distance is at least its counterpart here: when this sum exceeds r2, so does p's, and no
// subtree that could hold a match is skipped. (Binary32 keeps the test off the binary64 pipe,
// which runs at a small fraction of the binary32 rate on this GPU.)
__device__ __forceinline__ bool kt_may_hit(const float4* __restrict__ box, uint32_t m, float qx, float qy, float qz,
                                           float r2)
{
    const float4 lo = box[2 * m], hi = box[2 * m + 1];
    auto gap = [](float q, float l, float h) -> float { return (q < l) ? (l - q) : ((q > h) ? (q - h) : 0.0f); };
    const float gx = gap(qx, lo.x, hi.x), gy = gap(qy, lo.y, hi.y), gz = gap(qz, lo.z, hi.z);
    return (gx * gx) + ((gy * gy) + (gz * gz)) <= r2;
}

__device__ __forceinline__ int kt_scan_of(const BatchDev& b, uint32_t i)
{
    return scan_of_point(b, i); // (src_off == pt_off)
}

// Pool allocation of `count` entries, one atomic per group of converged lanes (the lanes loop
// over the group's members alike, so every shuffle has all of them); kNone when the pool is full.
__device__ __forceinline__ uint32_t kt_pool_alloc(uint32_t* head, uint32_t cap, uint32_t count)
{
    const uint32_t active = __activemask();
    const uint32_t lane = lane_id();
    uint32_t pre = 0, total = 0;
    for (uint32_t l = 0; l < 32; ++l)
        if ((active >> l) & 1u)
        {
            const uint32_t c = __shfl_sync(active, count, l);
            total += c;
            if (l < lane)
                pre += c;
        }
    const uint32_t leader = static_cast<uint32_t>(__ffs(static_cast<int>(active)) - 1);
    uint32_t base = 0;
    if (lane == leader && total)
        base = atomicAdd(head, total);
    base = __shfl_sync(active, base, leader);
    if (base > cap || cap - base < total)
        return kNone;
    return base + pre;
}

// Step 2: every point's own search; VALID points' leftovers into the pool. Thread t takes the
// point at tree position t (its input index from the build), so the threads of a warp query
// neighbouring points, whose searches walk largely the same nodes (cache hits, little divergence,
// where input order may be shuffled); the results go to the point's input index.
__global__ void k_kt_own(BatchDev b)
{
    pdl_enter();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= b.nsrc)
        return;
    const int s = kt_scan_of(b, t);
    const ScanDev& sd = b.scans[s];
    const float4 q = b.kt[t]; // the point's coordinates, as loaded from the input
    const uint32_t i = b.kq[t];
    if (i - sd.src_off >= sd.n_src)
    {
        raise_err(&b.state[s], ERR_INTERNAL); // not a point of this scan: reported, never followed
        return;
    }
    const float r2 = kt_radius2(sd, q);
    uint32_t stk[kKtStack];
    int sp = 0;
    bool overflow = false;
    stk[sp++] = kt_entry(sd.n_src / 2, 0);
    const float4* g = b.kt + sd.src_off;
    const uint32_t k = sd.dror_k;
    const uint32_t found = kt_search(g, sd.n_src, q.x, q.y, q.z, r2, k, 0, stk, sp, overflow);
    if (overflow)
        raise_err(&b.state[s], ERR_INTERNAL);
    const bool valid = found >= k;
    b.kown[i] = found;
    b.kshort[i] = valid ? 0u : 1u;
    uint32_t nleft = valid ? static_cast<uint32_t>(sp) : 0u;
    const uint32_t at = kt_pool_alloc(b.kctr, b.kpool_cap, nleft);
    if (at == kNone)
    {
        raise_err(&b.state[s], ERR_HASH_FULL); // leftover pool full: reported, scan invalid
        nleft = 0;
    }
    b.klo_n[i] = nleft;
    b.klo_at[i] = (at == kNone) ? 0u : at;
    for (uint32_t t = 0; t < nleft; ++t)
        b.kpool[at + t] = stk[t];
    if (valid)
        b.noise[i] = LP_NOISE_VALID;
}

// Leftovers into one array in point order (klo_off: exclusive scan of the counts).
__global__ void k_kt_flat(BatchDev b)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.nsrc)
        return;
    const uint32_t n = b.klo_off[i + 1] - b.klo_off[i];
    const uint32_t at = b.klo_at[i], to = b.klo_off[i];
    for (uint32_t t = 0; t < n; ++t)
        b.kflat[to + t] = b.kpool[at + t];
}

// The short points in order (kshort: exclusive scan of the flags).
__global__ void k_kt_short(BatchDev b)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.nsrc)
        return;
    if (b.kshort[i + 1] != b.kshort[i])
        b.kq[b.kshort[i]] = i;
}

// First entry (flat index) of the piece a short point meets on top of the stack: the leftovers of
// the points after the previous short point of its scan.
// The same for short point u once k_kt_segment has run: it records its piece's first entry in
// klo_n, which holds nothing else by then (one load instead of three dependent ones).
__device__ __forceinline__ uint32_t kt_piece_lo(const BatchDev& b, uint32_t u)
{
    return b.klo_n[u];
}

__device__ __forceinline__ uint32_t kt_segment_lo(const BatchDev& b, const ScanDev& sd, uint32_t t)
{
    const uint32_t first = b.kshort[sd.src_off];
    const uint32_t prev = (t > first) ? b.kq[t - 1] + 1 : sd.src_off;
    return b.klo_off[prev];
}

// A query through the piece arr[lo, hi) from the top (entries hi - 1 down), by a warp: 32 entries at a
// time are tested and, where their box is within the radius, searched in full, each from count 0;
// an ordered prefix of the counts finds the stop, whose search runs again from the count before it
// for what it leaves (into the pool). `found` counts on; returns whether it reached k, with the stop.
// (One thread per query took a piece's entries one after the other, a chain of dependent loads as
// long as the piece: 285 us for the 6,800 short points of a cloud of 110k, 545 us for 50,000 of 1M.)
struct KtStopAt
{
    uint32_t x, at, n; // the entry, and what its search left in the pool
};

__device__ __forceinline__ bool kt_walk_piece(const BatchDev& b, const ScanDev& sd, const uint32_t* arr, uint32_t lo, uint32_t hi,
                                              float4 q, float r2, uint32_t& found, KtStopAt& stop, uint32_t* stk, bool& overflow,
                                              bool& pool_full)
{
    const uint32_t lane = lane_id();
    const float4* g = b.kt + sd.src_off;
    const float4* box = b.kbb + 2ull * sd.src_off;
    const uint32_t k = sd.dror_k;
    for (uint32_t x = hi; x > lo; x -= min(32u, x - lo))
    {
        uint32_t e = 0u, cnt = 0u;
        bool near = false;
        if (lane < x - lo)
        {
            e = arr[x - 1u - lane];
            near = kt_may_hit(box, e >> 2, q.x, q.y, q.z, r2);
        }
        if (!__any_sync(0xffffffffu, near))
            continue;
        if (near)
        {
            int sp = 0;
            stk[sp++] = e;
            cnt = kt_search(g, sd.n_src, q.x, q.y, q.z, r2, k, 0, stk, sp, overflow);
        }
        __syncwarp();
        const uint32_t incl = warp_incl_scan(cnt);
        const uint32_t reach = __ballot_sync(0xffffffffu, cnt > 0u && found + incl >= k);
        if (reach != 0u)
        {
            const uint32_t hl = static_cast<uint32_t>(__ffs(static_cast<int>(reach)) - 1);
            uint32_t at = 0u, n = 0u;
            if (lane == hl)
            {
                int sp = 0;
                stk[sp++] = e;
                kt_search(g, sd.n_src, q.x, q.y, q.z, r2, k, found + incl - cnt, stk, sp, overflow);
                n = static_cast<uint32_t>(sp);
                at = n ? atomicAdd(b.kctr, n) : 0u;
                if (at > b.kpool_cap || b.kpool_cap - at < n)
                {
                    pool_full = true;
                    at = 0u;
                    n = 0u;
                }
                for (uint32_t u = 0; u < n; ++u)
                    b.kpool[at + u] = stk[u];
            }
            __syncwarp();
            stop = KtStopAt{x - 1u - hl, __shfl_sync(0xffffffffu, at, static_cast<int>(hl)),
                            __shfl_sync(0xffffffffu, n, static_cast<int>(hl))};
            found = k;
            return true;
        }
        found += __shfl_sync(0xffffffffu, incl, 31);
    }
    return false;
}

// Step 3: each short point through its own piece, a warp per point.
__global__ void k_kt_segment(BatchDev b)
{
    pdl_enter();
    const uint32_t lane = lane_id();
    const uint32_t nshort = b.kshort[b.nsrc];
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nshort; t += (gridDim.x * blockDim.x) >> 5)
    {
        const uint32_t i = b.kq[t];
        const int s = kt_scan_of(b, i);
        const ScanDev& sd = b.scans[s];
        const float4 q = b.src[i];
        const float r2 = kt_radius2(sd, q);
        uint32_t found = b.kown[i];
        const uint32_t lo = kt_segment_lo(b, sd, t), hi = b.klo_off[i];
        uint32_t stk[kKtStack];
        bool overflow = false, pool_full = false;
        KtStopAt stop{kNone, 0u, 0u};
        const bool hit = kt_walk_piece(b, sd, b.kflat, lo, hi, q, r2, found, stop, stk, overflow, pool_full);
        if (overflow)
            raise_err(&b.state[s], ERR_INTERNAL);
        if (pool_full)
            raise_err(&b.state[s], ERR_HASH_FULL);
        if (lane == 0)
        {
            b.klo_n[t] = lo; // for the candidate walks and the chain (klo_n is no longer read as counts)
            b.kc[t] = make_uint4(found, hit ? stop.x : kNone, stop.at, stop.n); // count, stop entry, left entries
            if (hit)
                b.noise[i] = LP_NOISE_VALID;
        }
    }
}

// Candidates: short points not decided in their own piece (flag -> exclusive scan -> list).
__global__ void k_kt_cand_flag(BatchDev b)
{
    pdl_enter();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nshort = b.kshort[b.nsrc];
    if (t == 0)
        b.kcflag[nshort] = 0;
    if (t < nshort)
        b.kcflag[t] = (b.kc[t].y == kNone) ? 1u : 0u;
}

__global__ void k_kt_cand_list(BatchDev b)
{
    pdl_enter();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < b.kshort[b.nsrc] && b.kcflag[t + 1] != b.kcflag[t])
        b.kcand[b.kcflag[t]] = t;
}

// Step 4a: every candidate walks the pieces pushed since the previous candidate, as if nothing
// lay below them (true when the previous candidate exhausted the stack): the pieces the short points
// since then pushed (all decided in their own piece: the rest of their piece below the stop, then the
// entries the stopping search left, on top), newest first. A warp per candidate.
__global__ void k_kt_spec(BatchDev b)
{
    pdl_enter();
    const uint32_t lane = lane_id();
    const uint32_t ncand = b.kcflag[b.kshort[b.nsrc]];
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < ncand; c += (gridDim.x * blockDim.x) >> 5)
    {
        const uint32_t t = b.kcand[c];
        const uint32_t i = b.kq[t];
        const int s = kt_scan_of(b, i);
        const ScanDev& sd = b.scans[s];
        const uint32_t t_first = b.kshort[sd.src_off];
        const uint32_t c_first = b.kcflag[t_first];
        const uint32_t tp1 = (c > c_first) ? b.kcand[c - 1] + 1 : t_first; // first pushing short point
        const float4 q = b.src[i];
        const float r2 = kt_radius2(sd, q);
        uint32_t found = b.kc[t].x;
        uint32_t stk[kKtStack];
        bool overflow = false, pool_full = false, hit = false;
        KtStopAt stop{0u, 0u, 0u};
        uint32_t hu = kNone, hkind = 0u;
        for (uint32_t u = t; !hit && u > tp1;)
        {
            --u;
            const uint4 cu = b.kc[u];
            hkind = 1u;
            hit = kt_walk_piece(b, sd, b.kpool, cu.z, cu.z + cu.w, q, r2, found, stop, stk, overflow, pool_full);
            if (!hit)
            {
                hkind = 0u;
                hit = kt_walk_piece(b, sd, b.kflat, kt_piece_lo(b, u), cu.y, q, r2, found, stop, stk, overflow, pool_full);
            }
            hu = u;
        }
        if (overflow)
            raise_err(&b.state[s], ERR_INTERNAL);
        if (pool_full)
            raise_err(&b.state[s], ERR_HASH_FULL);
        if (lane == 0)
        {
            b.kspec[c] = hit ? make_uint4(found, hu, stop.x | (hkind << 31), stop.at) : make_uint4(found, kNone, 0u, 0u);
            b.kspec_n[c] = hit ? stop.n : 0u;
            // the result unless the candidate reaches the count in what lies below (k_kt_run, k_kt_chain)
            b.noise[i] = hit ? LP_NOISE_VALID : LP_NOISE_NOISE;
        }
    }
}

// Record of a candidate's walk through what its predecessor's stop left (k_kt_spec_next), in
// arrays free by then (per candidate c): kscr[2c] stop entry, kscr[2c + 1] where the entries that
// stopping search left start in the pool, kown[c] count, klo_at[c] = status | left count << 2 |
// piece << 9 (the stop's piece, counted from the top of those pieces).
constexpr uint32_t kNextNone = 0u, kNextStop = 1u, kNextOut = 2u;
constexpr uint32_t kNextPieceMax = 1u << 23;

// Step 4a': a candidate whose walk ran out, right after a candidate whose walk stopped, continues
// into R, and R is then what it was before that stop with the stop's pieces on top: the pieces of
// the predecessor's pushing points below its stop point u, the rest of u's pieces below the stop,
// and the entries the stopping search left (the chain pushes exactly these, in this order). Every
// such candidate walks those pieces here, in parallel, from its count after its own walk. The
// chain takes the result when the predecessor's stop is the last change to R: a stop in those
// pieces is exact whatever lies below them; running out of them continues into R below.
__global__ void k_kt_spec_next(BatchDev b)
{
    pdl_enter();
    const uint32_t lane = lane_id();
    const uint32_t ncand = b.kcflag[b.kshort[b.nsrc]];
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < ncand; c += (gridDim.x * blockDim.x) >> 5)
    {
        uint32_t status = kNextNone, piece = 0u, found = 0u;
        KtStopAt stop{0u, 0u, 0u};
        const uint32_t t = b.kcand[c];
        const uint32_t i = b.kq[t];
        const int s = kt_scan_of(b, i);
        const ScanDev& sd = b.scans[s];
        const uint32_t t_first = b.kshort[sd.src_off];
        const uint32_t c_first = b.kcflag[t_first];
        // the scan's first candidate has no predecessor
        const uint4 own = b.kspec[c], pv = (c == c_first) ? make_uint4(0u, kNone, 0u, 0u) : b.kspec[c - 1];
        if (own.y == kNone && pv.y != kNone) // this walk ran out, the predecessor's stopped
        {
            const uint32_t tp1 = (c - 1 > c_first) ? b.kcand[c - 2] + 1 : t_first; // the predecessor's first pushing point
            const uint32_t hu = pv.y, hx = pv.z & 0x7fffffffu, hkind = pv.z >> 31;
            const float4 q = b.src[i];
            const float r2 = kt_radius2(sd, q);
            found = own.x;
            uint32_t stk[kKtStack];
            bool overflow = false, pool_full = false;
            // one piece; an empty piece is not in R and is not counted
            auto walk = [&](uint32_t lo, uint32_t hi, const uint32_t* arr) -> bool {
                if (hi <= lo)
                    return false;
                if (kt_walk_piece(b, sd, arr, lo, hi, q, r2, found, stop, stk, overflow, pool_full))
                    return true;
                ++piece;
                return false;
            };
            bool stopped = walk(pv.w, pv.w + b.kspec_n[c - 1], b.kpool);
            if (!stopped)
            {
                const uint4 cu = b.kc[hu];
                if (hkind == 1)
                    stopped = walk(cu.z, hx, b.kpool) || walk(kt_piece_lo(b, hu), cu.y, b.kflat);
                else
                    stopped = walk(kt_piece_lo(b, hu), hx, b.kflat);
            }
            for (uint32_t u = hu; !stopped && u > tp1;)
            {
                --u;
                const uint4 cu = b.kc[u];
                stopped = walk(cu.z, cu.z + cu.w, b.kpool) || walk(kt_piece_lo(b, u), cu.y, b.kflat);
            }
            if (overflow)
                raise_err(&b.state[s], ERR_INTERNAL);
            if (pool_full)
                raise_err(&b.state[s], ERR_HASH_FULL);
            if (piece < kNextPieceMax && !__any_sync(0xffffffffu, overflow || pool_full))
                status = stopped ? kNextStop : kNextOut; // (else the run searches the pieces itself)
        }
        if (lane == 0)
        {
            if (status != kNextNone)
            {
                b.kscr[2ull * c] = stop.x;
                b.kscr[2ull * c + 1] = stop.at;
                b.kown[c] = found;
            }
            b.klo_at[c] = status | (stop.n << 2) | (piece << 9);
        }
        __syncwarp();
    }
}

// Step 4b: the stopped candidates of the batch in order (kstop).
struct StopSrc
{
    BatchDev b;
    __device__ __forceinline__ uint32_t count() const { return b.kcflag[b.kshort[b.nsrc]]; }
    __device__ __forceinline__ uint32_t end() const { return count() + 1u; }
    __device__ __forceinline__ uint4 get4(uint32_t i) const
    {
        const uint32_t n = count();
        auto one = [&](uint32_t c) { return (c < n && b.kspec[c].y != kNone) ? 1u : 0u; };
        return make_uint4(one(i), one(i + 1u), one(i + 2u), one(i + 3u));
    }
};
struct StopDst
{
    BatchDev b;
    __device__ __forceinline__ void put4(uint32_t i, uint4 e, uint4 f) const
    {
        if (f.x)
            b.kstop[e.x] = i;
        if (f.y)
            b.kstop[e.y] = i + 1u;
        if (f.z)
            b.kstop[e.z] = i + 2u;
        if (f.w)
            b.kstop[e.w] = i + 3u;
        const uint32_t n = b.kcflag[b.kshort[b.nsrc]];
        if (i <= n && n < i + 4u) // the count, from the entry past the last candidate
            b.kctr[1] = (n == i) ? e.x : ((n == i + 1u) ? e.y : ((n == i + 2u) ? e.z : e.w));
    }
};

// A stack of pieces (lo, hi): entries [lo, hi) of the flat array (bit 31 of lo clear) or of the pool
// (set), consumed from hi - 1 down. Control flow is uniform over the CTA: every thread holds the same
// top, count and candidate; thread 0 writes the stack and the pool, and a barrier precedes every read.
constexpr uint32_t kChainThreads = 256;
constexpr uint32_t kChainPieces = 32;

struct ChainShared
{
    uint32_t red[kChainThreads / 32];
    uint32_t bc[4];
    uint2 pc[kChainPieces]; // the top pieces of the stack for one round (index 0 = the top)
    uint32_t pre[kChainPieces + 1]; // and their entry-count prefix
};

struct ChainStack
{
    uint2* R;
    uint32_t cap, top;
    bool overflow, pool_full, full;
    __device__ __forceinline__ void push(uint32_t lo, uint32_t hi)
    {
        if (hi > (lo & 0x7fffffffu))
        {
            if (top < cap)
            {
                if (threadIdx.x == 0)
                    R[top] = make_uint2(lo, hi);
                ++top;
            }
            else
                full = true;
        }
    }
};

// block-wide minimum and inclusive sum (every thread gets the result)
__device__ __forceinline__ uint32_t chain_min(uint32_t* red, uint32_t v)
{
    v = __reduce_min_sync(0xffffffffu, v);
    if (lane_id() == 0)
        red[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t m = red[0];
#pragma unroll
    for (uint32_t w = 1; w < kChainThreads / 32u; ++w)
        m = min(m, red[w]);
    __syncthreads();
    return m;
}
__device__ __forceinline__ uint32_t chain_incl(uint32_t* red, uint32_t v, uint32_t& total)
{
    v = warp_incl_scan(v);
    if (lane_id() == 31)
        red[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t pre = 0;
    total = 0;
#pragma unroll
    for (uint32_t w = 0; w < kChainThreads / 32u; ++w)
    {
        const uint32_t x = red[w];
        if (w < (threadIdx.x >> 5))
            pre += x;
        total += x;
    }
    __syncthreads();
    return v + pre;
}

// A candidate continues into the stack from count `found`: up to kChainThreads entries at a time across
// the top kChainPieces pieces; every thread searches one entry's subtree in full (these searches,
// chains of dependent node loads, are the cost, so a round is as wide as the CTA), and an ordered
// prefix of the counts finds the stop. True: the count was reached, and the stack holds what that
// leaves; false: the stack is empty.
__device__ bool chain_search(const BatchDev& b, const ScanDev& sd, ChainStack& S, ChainShared& sh, float4 q, uint32_t& found,
                             uint32_t* stk)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const float4* g = b.kt + sd.src_off;
    const float4* box = b.kbb + 2ull * sd.src_off;
    const uint32_t k = sd.dror_k;
    const float r2 = kt_radius2(sd, q);
    while (S.top > 0)
    {
        // the top pieces (warp 0) and how many entries of them this round covers
        const uint32_t np = min(S.top, kChainPieces);
        if (warp == 0)
        {
            const uint2 pc = (lane < np) ? S.R[S.top - 1 - lane] : make_uint2(0u, 0u);
            const uint32_t sz = (lane < np) ? pc.y - (pc.x & 0x7fffffffu) : 0u;
            const uint32_t incl = warp_incl_scan(sz);
            if (lane < np)
                sh.pc[lane] = pc;
            sh.pre[lane + 1] = incl;
            if (lane == 0)
                sh.pre[0] = 0;
        }
        __syncthreads();
        const uint32_t covered = min(sh.pre[np], kChainThreads);
        uint32_t cnt = 0, my_p = 0;
        if (tid < covered)
        {
            // the piece holding this thread's entry: the last p with pre[p] <= tid
            uint32_t lo_p = 0, hi_p = np - 1;
            while (lo_p < hi_p)
            {
                const uint32_t mid = (lo_p + hi_p + 1) / 2;
                if (sh.pre[mid] <= tid)
                    lo_p = mid;
                else
                    hi_p = mid - 1;
            }
            my_p = lo_p;
            const uint2 pc = sh.pc[my_p];
            const uint32_t* arr = (pc.x & 0x80000000u) ? b.kpool : b.kflat;
            const uint32_t e = arr[pc.y - 1 - (tid - sh.pre[my_p])];
            if (kt_may_hit(box, e >> 2, q.x, q.y, q.z, r2))
            {
                int sp = 0;
                stk[sp++] = e;
                cnt = kt_search(g, sd.n_src, q.x, q.y, q.z, r2, k, 0, stk, sp, S.overflow);
            }
        }
        uint32_t total = 0;
        const uint32_t incl = chain_incl(sh.red, cnt, total);
        if (total > 0 && found + total >= k)
        {
            const uint32_t hl = chain_min(sh.red, (tid < covered && cnt > 0 && found + incl >= k) ? tid : kNone);
            if (tid == hl)
            {
                sh.bc[0] = found + incl - cnt; // the count before the stopping entry
                sh.bc[3] = my_p;
            }
            __syncthreads();
            const uint32_t before = sh.bc[0], p = sh.bc[3];
            const uint2 pc = sh.pc[p];
            const uint32_t x = pc.y - 1 - (hl - sh.pre[p]);
            const uint32_t* arr = (pc.x & 0x80000000u) ? b.kpool : b.kflat;
            // the stopping search again on thread 0, from the count before it, for what it leaves
            if (tid == 0)
            {
                int sp = 0;
                stk[sp++] = arr[x];
                kt_search(g, sd.n_src, q.x, q.y, q.z, r2, k, before, stk, sp, S.overflow);
                uint32_t at = kt_pool_alloc(b.kctr, b.kpool_cap, static_cast<uint32_t>(sp));
                if (at == kNone)
                {
                    S.pool_full = true;
                    at = 0;
                    sp = 0;
                }
                for (int v = 0; v < sp; ++v)
                    b.kpool[at + v] = stk[v];
                sh.bc[1] = static_cast<uint32_t>(sp);
                sh.bc[2] = at;
            }
            __syncthreads();
            const uint32_t nsp = sh.bc[1], at = sh.bc[2];
            // the pieces above p are consumed, p keeps its entries below the stop, then the left
            // entries go on top
            S.top -= p + 1;
            S.push(pc.x, x);
            S.push(at | 0x80000000u, at + nsp);
            __syncthreads();
            return true;
        }
        found += total;
        // pieces fully covered are consumed; the last covered one keeps what lies below
        uint32_t p = 0;
        while (p < np && sh.pre[p + 1] <= covered)
            ++p;
        S.top -= p;
        if (p < np && covered > sh.pre[p] && tid == 0)
            S.R[S.top - 1].y = sh.pc[p].y - (covered - sh.pre[p]);
        __syncthreads();
    }
    return false;
}

__device__ __forceinline__ void chain_report(ScanState* st, const ChainStack& S)
{
    if (__syncthreads_or(S.overflow) && threadIdx.x == 0)
        raise_err(st, ERR_INTERNAL);
    if (__syncthreads_or(S.pool_full) && threadIdx.x == 0)
        raise_err(st, ERR_HASH_FULL);
    if (S.full && threadIdx.x == 0)
        raise_err(st, ERR_INTERNAL);
}

// Step 4c: runs. A run is a candidate whose walk stopped and the candidates after it, whose walks ran
// out, up to the next that stopped: the stop's remainder goes onto the stack, and each of the others
// continues into the stack until one empties it; from there to the end of the run the candidates are
// NOISE. As if nothing lay below the run's own pieces, the runs are independent, one CTA each; only
// one run in twenty meets a stack that is not empty (k_kt_chain puts those right), where one
// CTA per scan taking all candidates in order spent 5.6 ms on a cloud of 1M points.
//
// Run j's pieces lie in kpiece from twice the scan-local index of its first pushing short point: every
// short point of a run adds at most two pieces. Its result replaces the stop's record: (the candidate
// that emptied the run's pieces or kNone, its count then, pieces left, their place in kpiece).
__global__ void __launch_bounds__(kChainThreads) k_kt_run(BatchDev b)
{
    pdl_enter();
    __shared__ ChainShared sh;
    const uint32_t tid = threadIdx.x;
    const uint32_t nstop = b.kctr[1];
    uint32_t stk[kKtStack];
    for (uint32_t j = blockIdx.x; j < nstop; j += gridDim.x)
    {
        const uint32_t c = b.kstop[j];
        const uint32_t i = b.kq[b.kcand[c]];
        const int s = kt_scan_of(b, i);
        const ScanDev& sd = b.scans[s];
        const uint32_t t_first = b.kshort[sd.src_off];
        const uint32_t c0 = b.kcflag[t_first], c1 = b.kcflag[b.kshort[sd.src_off + sd.n_src]];
        const uint32_t end = (j + 1u < nstop) ? min(b.kstop[j + 1u], c1) : c1;
        const uint32_t tp1 = (c > c0) ? b.kcand[c - 1u] + 1u : t_first;
        const uint32_t base = 2u * (tp1 - t_first);
        ChainStack S{b.kpiece + 2ull * sd.src_off + 2ull * static_cast<uint32_t>(s) + base, 2u * (b.kcand[end - 1u] + 1u - tp1), 0u,
                     false, false, false};
        // the stop: the pieces of the pushing points below the stop point, then the rest of that
        // point's pieces below the stop, then the entries the stopping search left
        const uint4 rec = b.kspec[c];
        const uint32_t hu = rec.y, hx = rec.z & 0x7fffffffu, hkind = rec.z >> 31;
        for (uint32_t u = tp1; u <= hu; ++u)
        {
            const uint4 cu = b.kc[u];
            const uint32_t lo = kt_piece_lo(b, u);
            if (u < hu)
            {
                S.push(lo, cu.y);
                S.push(cu.z | 0x80000000u, cu.z + cu.w);
            }
            else if (hkind == 1)
            {
                S.push(lo, cu.y);
                S.push(cu.z | 0x80000000u, hx);
            }
            else
            {
                S.push(lo, hx);
            }
        }
        S.push(rec.w | 0x80000000u, rec.w + b.kspec_n[c]);
        __syncthreads(); // thread 0's pieces are read by every thread next
        uint32_t out = kNone, count = 0u;
        for (uint32_t x = c + 1u; x < end; ++x)
        {
            const uint32_t xi = b.kq[b.kcand[x]];
            uint32_t found = b.kspec[x].x;
            bool hit = false;
            if (x == c + 1u)
            {
                // its walk through the stop's pieces is done (k_kt_spec_next)
                const uint32_t w = b.klo_at[x];
                const uint32_t status = w & 3u, nsp = (w >> 2) & 127u, p = w >> 9;
                if (status == kNextStop && p < S.top)
                {
                    const uint32_t sx = b.kscr[2ull * x], sat = b.kscr[2ull * x + 1u];
                    const uint2 pc = S.R[S.top - 1u - p];
                    __syncthreads();
                    S.top -= p + 1u;
                    S.push(pc.x, sx);
                    S.push(sat | 0x80000000u, sat + nsp);
                    __syncthreads();
                    hit = true;
                }
                else if (status == kNextOut)
                {
                    found = b.kown[x];
                    S.top = 0u;
                }
            }
            if (!hit)
                hit = chain_search(b, sd, S, sh, b.src[xi], found, stk);
            if (!hit)
            {
                out = x;
                count = found;
                break;
            }
            if (tid == 0)
                b.noise[xi] = LP_NOISE_VALID;
        }
        if (tid == 0)
            b.kspec[c] = make_uint4(out, count, S.top, base);
        chain_report(&b.state[s], S);
    }
}

// Step 4d: one CTA per scan takes the runs in order with what earlier runs left (the stack at the front
// of the scan's kpiece: it never reaches the pieces of the run at hand). While the stack is empty,
// runs that left nothing stand as they are; a run that emptied its own pieces above a stack that is not
// empty continues into it from the candidate that did.
__global__ void __launch_bounds__(kChainThreads) k_kt_chain(BatchDev b)
{
    pdl_enter();
    __shared__ ChainShared sh;
    const int s = blockIdx.x;
    const ScanDev& sd = b.scans[s];
    const uint32_t tid = threadIdx.x;
    const uint32_t c0 = b.kcflag[b.kshort[sd.src_off]], c1 = b.kcflag[b.kshort[sd.src_off + sd.n_src]];
    const uint32_t nstop = b.kctr[1];
    // the scan's runs [j, j1): the first stops at or after c0 and c1
    uint32_t j1 = 0u, j = 0u;
    for (uint32_t step = 1u << 31; step != 0u; step >>= 1)
    {
        if (j + step <= nstop && b.kstop[j + step - 1u] < c0)
            j += step;
        if (j1 + step <= nstop && b.kstop[j1 + step - 1u] < c1)
            j1 += step;
    }
    uint2* R = b.kpiece + 2ull * sd.src_off + 2ull * static_cast<uint32_t>(s);
    ChainStack S{R, 2u * sd.n_src + 2u, 0u, false, false, false};
    uint32_t stk[kKtStack];
    while (j < j1)
    {
        if (S.top == 0u)
        {
            // on to the next run that left pieces
            const uint32_t jj = j + tid;
            const bool left = jj < j1 && b.kspec[b.kstop[jj]].z != 0u;
            const uint32_t h = chain_min(sh.red, left ? tid : kNone);
            j += (h == kNone) ? kChainThreads : h;
            if (h == kNone)
                continue;
        }
        const uint32_t c = b.kstop[j];
        const uint4 run = b.kspec[c];
        ++j;
        if (run.z != 0u)
        {
            // its pieces on top of the stack (they move down: every chunk is read before it is written)
            for (uint32_t k0 = 0; k0 < run.z; k0 += kChainThreads)
            {
                uint2 v = make_uint2(0u, 0u);
                if (k0 + tid < run.z)
                    v = R[run.w + k0 + tid];
                __syncthreads();
                if (k0 + tid < run.z)
                    R[S.top + k0 + tid] = v;
                __syncthreads();
            }
            S.top += run.z;
            continue;
        }
        if (run.x == kNone)
            continue;
        const uint32_t end = (j < j1) ? b.kstop[j] : c1;
        for (uint32_t x = run.x; x < end && S.top > 0u; ++x)
        {
            const uint32_t xi = b.kq[b.kcand[x]];
            uint32_t found = (x == run.x) ? run.y : b.kspec[x].x;
            if (chain_search(b, sd, S, sh, b.src[xi], found, stk) && tid == 0)
                b.noise[xi] = LP_NOISE_VALID;
        }
    }
    chain_report(&b.state[s], S);
}
} // namespace

size_t kt_build_smem_bytes()
{
    // a subtree's records, then two uint16 candidate lists per point
    return static_cast<size_t>(kKtSmall) * sizeof(float4) + static_cast<size_t>(kKtSmall) * 2 * sizeof(uint16_t);
}
size_t kt_stage_smem_bytes()
{
    return static_cast<size_t>(kKtStage) * sizeof(float4) + static_cast<size_t>(kKtStage) * 2 * sizeof(uint16_t);
}

void init_kdtree_attributes()
{
    cudaFuncSetAttribute(k_kt_level, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kt_stage_smem_bytes()));
    cudaFuncSetAttribute(k_kt_level_huge, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kt_stage_smem_bytes()));
    cudaFuncSetAttribute(k_kt_small, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kt_build_smem_bytes()));
}

void launch_noise(Launcher& L, const BatchDev& b, const BatchHost& hb, const lp_noise_remover_config& cfg)
{
    (void)cfg;
    const uint32_t T = 256;
    uint32_t nmax = 0;
    for (const ScanDev& sd : hb.scans)
        nmax = std::max(nmax, sd.n_src);
    if (nmax == 0)
        return;
    LP_LAUNCH(L, k_kt_load, div_up(b.nsrc, T), T, b);
    // levels until every range of the deepest level is at most kKtSmall (then built in shared memory)
    int levels = 1;
    while ((nmax >> (levels - 1)) > kKtSmall)
        ++levels;
    const uint32_t S = static_cast<uint32_t>(b.nscan);
    for (int l = 0; l < levels; ++l)
    {
        const uint32_t slots = 1u << l;
        // a level of few ranges leaves SMs idle with one CTA each: clusters take smaller ranges too
        const uint32_t huge = (S * slots * kKtCluster <= static_cast<uint32_t>(sm_count())) ? kKtFew : kKtHuge;
        if ((nmax >> l) > huge)
            LP_LAUNCH_SMEM(L, k_kt_level_huge, S * slots * kKtCluster, kKtThreads, kt_stage_smem_bytes(), b, l, slots, huge);
        // a scan's longest range on the level has n >> l points, its shortest ((n + 1) >> l) - 1
        bool mid = false, small = false;
        for (const ScanDev& sd : hb.scans)
        {
            const uint32_t longest = sd.n_src >> l, shortest = ((sd.n_src + 1u) >> l) - (((sd.n_src + 1u) >> l) ? 1u : 0u);
            mid |= longest > kKtSmall && shortest <= huge;
            small |= shortest <= kKtSmall && (l == 0 || (sd.n_src >> (l - 1)) > kKtSmall);
        }
        if (mid)
            LP_LAUNCH_SMEM(L, k_kt_level, S * slots, kKtThreads, kt_stage_smem_bytes(), b, l, slots, huge);
        if (small) // wide CTAs finish a subtree sooner, narrow ones share an SM better
            LP_LAUNCH_SMEM(L, k_kt_small, S * slots, (S * slots <= static_cast<uint32_t>(sm_count()) * 2u) ? kKtSmallThreads : kKtSmallThreads / 2,
                           kt_build_smem_bytes(), b, l, slots);
    }
    for (int l = levels - 2; l >= 0; --l)
    {
        const uint32_t slots = 1u << l;
        LP_LAUNCH(L, k_kt_box_level, div_up(S * slots, 128u), 128, b, l, slots);
    }
    LP_LAUNCH(L, k_kt_own, div_up(b.nsrc, 128u), 128, b);
    L.scan(b.klo_n, b.klo_off, b.nsrc + 1);
    L.scan(b.kshort, b.kshort, b.nsrc + 1);
    LP_LAUNCH(L, k_kt_flat, div_up(b.nsrc, T), T, b);
    LP_LAUNCH(L, k_kt_short, div_up(b.nsrc, T), T, b);
    // a warp per short point or candidate: grid-strided (few of the points are)
    const uint32_t wgrid = std::min(div_up(b.nsrc, 8u), static_cast<uint32_t>(sm_count()) * 8u);
    LP_LAUNCH(L, k_kt_segment, wgrid, 256, b);
    LP_LAUNCH(L, k_kt_cand_flag, div_up(b.nsrc + 1, T), T, b);
    L.scan(b.kcflag, b.kcflag, b.nsrc + 1);
    LP_LAUNCH(L, k_kt_cand_list, div_up(b.nsrc, T), T, b);
    LP_LAUNCH(L, k_kt_spec, wgrid, 256, b);
    LP_LAUNCH(L, k_kt_spec_next, wgrid, 256, b);
    if (uint32_t* words = L.scan_state(b.nsrc + 1))
    {
        L.begin("k_kt_stops");
        scan_lookback(L.stream, StopSrc{b}, StopDst{b}, b.nsrc + 1, words, L.scan_err, true, L.overlap);
        L.end();
        L.note();
    }
    LP_LAUNCH(L, k_kt_run, std::min(b.nsrc, static_cast<uint32_t>(sm_count()) * 8u), kChainThreads, b);
    LP_LAUNCH(L, k_kt_chain, S, kChainThreads, b);
}
} // namespace lpg
