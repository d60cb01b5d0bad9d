// lp_segment.cu — ground segmentation kernels (ring partition, polar grid, RECM, RANSAC,
// range-image projection, dilation, jump convolution, label population).
//
// Reference: lidar_processing_lib/src/segmenter.cpp (Segmenter::segment and helpers) and
// src/dataloader/src/dataloader.cpp:68-137 (ring partition). Every binary32 expression keeps
// the reference's operation order; the library is compiled with --fmad=false so that no
// multiply-add is contracted.
#include <cfloat>

#include <mutex>
#include <random>

#include "lp_batch.cuh"
#include "lp_common.cuh"
#include "lp_math.cuh"
#include "lp_stages.hpp"

namespace lpg
{
namespace
{
constexpr float kPiF = 3.14159274101257324219f;       // M_PIf
constexpr float kPi2F = 1.57079637050628662109f;      // M_PI_2f
constexpr float kPi15F = 4.71238899230957031250f;     // 1.5F * M_PIf (dataloader.cpp:108)
constexpr float kTwoPiF = 6.28318548202514648438f;    // 2.0F * M_PIf == (float)(2*M_PI)
constexpr int kRingTile = 1024;
constexpr int kMediumCell = 256; // sorted in shared memory by one warp
constexpr uint32_t kLargeCellMax = 8192;

__device__ __forceinline__ int scan_of_pix(const BatchDev& b, uint32_t p)
{
    return b.nscan <= kFewScans ? b.pix_few.find(p) : find_scan(b.nscan, p, [&](int s) { return b.scans[s].pix_off; });
}
__device__ __forceinline__ int scan_of_row(const BatchDev& b, uint32_t r)
{
    return b.nscan <= kFewScans ? b.row_few.find(r) : find_scan(b.nscan, r, [&](int s) { return b.scans[s].row_off; });
}
__device__ __forceinline__ int scan_of_tile(const BatchDev& b, uint32_t t)
{
    return find_scan(b.nscan, t, [&](int s) { return b.scans[s].tile_off; });
}
__device__ __forceinline__ int scan_of_slice(const BatchDev& b, uint32_t t)
{
    return b.nscan <= kFewScans ? b.slice_few.find(t) : find_scan(b.nscan, t, [&](int s) { return b.scans[s].slice_off; });
}

// ------------------------------------------------------------------------------------------
// Ring partition (dataloader.cpp:68-137): quadrant of the wrapped azimuth, FOURTH->FIRST
// transitions counted by a prefix scan, ring = first_ring - min(first_ring, count).
// ------------------------------------------------------------------------------------------
__global__ void k_quadrant(BatchDev b)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.npts)
        return;
    const float4 p = b.pts[i];
    float az = lpm::cr_atan2f(p.y, p.x);
    az = (az < 0) ? (az + kTwoPiF) : az;
    uint8_t q;
    if (az < kPi2F)
        q = 0;
    else if (az < kPiF)
        q = 1;
    else if (az < kPi15F)
        q = 2;
    else
        q = 3;
    b.quad[i] = q;
}

__device__ __forceinline__ uint32_t ring_flag(const BatchDev& b, const ScanDev& sd, uint32_t i)
{
    // point i (global) starts a new ring: FIRST after FOURTH, not the scan's first point
    return (i > sd.pt_off && b.quad[i] == 0 && b.quad[i - 1] == 3) ? 1u : 0u;
}

__global__ void __launch_bounds__(256) k_ring_count(BatchDev b)
{
    pdl_enter();
    const uint32_t t = blockIdx.x;
    const int s = scan_of_tile(b, t);
    const ScanDev& sd = b.scans[s];
    const uint32_t first = sd.pt_off + (t - sd.tile_off) * kRingTile;
    const uint32_t end = sd.pt_off + b.state[s].n_pts;
    uint32_t c = 0;
    for (uint32_t k = threadIdx.x; k < kRingTile; k += blockDim.x)
    {
        const uint32_t i = first + k;
        if (i < end)
            c += ring_flag(b, sd, i);
    }
    c = warp_sum(c);
    __shared__ uint32_t sm[8];
    if (lane_id() == 0)
        sm[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        uint32_t tot = 0;
        for (int w = 0; w < 8; ++w)
            tot += sm[w];
        b.tile_cnt[t] = tot;
    }
}

// tile_cnt holds the exclusive scan of the per-tile counts over the whole batch.
__global__ void __launch_bounds__(256) k_ring_apply(BatchDev b)
{
    pdl_enter();
    __shared__ uint32_t sm[33];
    const uint32_t t = blockIdx.x;
    const int s = scan_of_tile(b, t);
    const ScanDev& sd = b.scans[s];
    const uint32_t first = sd.pt_off + (t - sd.tile_off) * kRingTile;
    const uint32_t end = sd.pt_off + b.state[s].n_pts;
    const uint32_t base = b.tile_cnt[t] - b.tile_cnt[sd.tile_off];
    // 4 consecutive points per thread keep the scan in point order
    const uint32_t i0 = first + threadIdx.x * 4;
    uint32_t f[4];
    uint32_t loc = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        f[k] = (i0 + k < end) ? ring_flag(b, sd, i0 + k) : 0u;
        loc += f[k];
    }
    uint32_t total;
    uint32_t pre = block_excl_scan(loc, sm, &total) + base;
    const uint32_t fr = static_cast<uint32_t>(sd.first_ring);
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        pre += f[k];
        if (i0 + k < end)
            b.ring[i0 + k] = static_cast<uint16_t>(fr - min(fr, pre));
    }
}

// ------------------------------------------------------------------------------------------
// Polar grid (constructPolarGrid, segmenter.cpp:103-204).
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ int32_t bin_point(const BatchDev& b, uint32_t i, const float4 p)
{
    const int s = scan_of_point(b, i);
    const ScanDev& sd = b.scans[s];
    if (i - sd.pt_off >= b.state[s].n_pts)
        return -1; // slot left empty by noise removal
    if (p.z < sd.zmin_adj || p.z > sd.zmax_adj)
        return -1;
    const float d = sqrtf(p.x * p.x + p.y * p.y);
    const int32_t radial = static_cast<int32_t>(d / sd.spacing);
    if (d < sd.min_d || d > sd.max_d || radial >= sd.nrad)
        return -1;
    float az = lpm::atan2_approx(p.y, p.x);
    az = (az < 0) ? (az + kTwoPiF) : az;
    const int32_t slice = min(static_cast<int32_t>(az / sd.slice_res), sd.nslice - 1);
    int32_t h;
    if (sd.use_ring)
    {
        h = b.ring[i];
        if (h >= sd.H)
            return -1;
    }
    else
    {
        const float el = lpm::cr_atanf(p.z / d);
        h = static_cast<int32_t>((el - sd.down_rad) / sd.rad_per_px);
        if (h < 0 || h >= sd.H)
            return -1;
    }
    const int32_t w = static_cast<int32_t>(static_cast<uint16_t>(static_cast<float>(sd.W - 1) * az / kTwoPiF));
    b.pt_pix[i] = h * sd.W + w;
    return static_cast<int32_t>(sd.cell_off + static_cast<uint32_t>(slice * sd.nrad + radial));
}

// Two points per thread (i and i + blockDim.x), both loaded before either is binned.
__global__ void k_bin(BatchDev b)
{
    pdl_enter();
    const uint32_t i0 = blockIdx.x * blockDim.x * 2u + threadIdx.x;
    const uint32_t i1 = i0 + blockDim.x;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 p0 = (i0 < b.npts) ? b.pts[i0] : z4;
    const float4 p1 = (i1 < b.npts) ? b.pts[i1] : z4;
    const int32_t c0 = (i0 < b.npts) ? bin_point(b, i0, p0) : -1;
    const int32_t c1 = (i1 < b.npts) ? bin_point(b, i1, p1) : -1;
    if (i0 < b.npts)
        b.pt_cell[i0] = c0;
    if (i1 < b.npts)
        b.pt_cell[i1] = c1;
    // slot of the point in its cell (the order within a cell is free)
    const uint32_t s0 = warp_aggregated_inc(b.cell_cnt, static_cast<uint32_t>(c0), c0 >= 0);
    const uint32_t s1 = warp_aggregated_inc(b.cell_cnt, static_cast<uint32_t>(c1), c1 >= 0);
    if (c0 >= 0)
        b.pt_slot[i0] = s0;
    if (c1 >= 0)
        b.pt_slot[i1] = s1;
}

// (the per-point loads are issued before the scan lookup and the branch, which they do not need)
__global__ void k_scatter(BatchDev b)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.npts)
        return;
    const int32_t c = b.pt_cell[i];
    const uint32_t slot = b.pt_slot[i];
    const float z = b.pts[i].z;
    if (c < 0)
        return;
    const int s = scan_of_point(b, i);
    const uint32_t pos = b.cell_start[c] + slot;
    b.csr_idx[pos] = static_cast<int32_t>(i - b.scans[s].pt_off);
    b.csr_z[pos] = z;
}

// zlow of a cell (segmenter.cpp:249-260): with the cell's heights sorted, z[k] for the largest k
// in [1, n/2] with z[k] - z[k-1] > 0.5, else z[0].
//
// No sort is needed for it. Heights fall into half-metre buckets [q/2, (q+1)/2) with
// q = floor(2z) (2z and floor are exact in binary32). Two heights of one bucket differ by less
// than 0.5, so their float difference is at most 0.5: a qualifying k can only be where the sorted
// order crosses from a non-empty bucket A to the next non-empty bucket B, with z[k] = min(B),
// z[k-1] = max(A) and k = the number of heights below B. A warp therefore accumulates count, min
// and max per bucket and evaluates exactly the reference's test at those boundaries. Cells whose
// heights leave the bucket range (a nan, a range over 16 m) take the sorting path.
__device__ __forceinline__ uint32_t zord(float f)
{
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float zunord(uint32_t u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ bool cell_zlow_hist(const BatchDev& b, const ScanDev& sd, uint32_t c, uint32_t n, uint32_t start)
{
    const uint32_t lane = lane_id();
    const int32_t q0 = static_cast<int32_t>(floorf(2.0f * sd.zmin_adj));
    const int32_t nb = static_cast<int32_t>(floorf(2.0f * sd.zmax_adj)) - q0 + 1;
    if (!(nb >= 1 && nb <= 32))
        return false;
    // lane q accumulates bucket q; each step of 32 heights is folded in once per distinct bucket
    // (ground cells hold one or two) with warp reductions instead of contended atomics
    uint32_t cnt = 0u, lo = 0xffffffffu, hi = 0u;
    bool bad = false;
    float znext = (lane < n) ? b.csr_z[start + lane] : 0.0f;
    for (uint32_t base = 0; base < n; base += 32)
    {
        const uint32_t k = base + lane;
        int32_t q = -1;
        uint32_t zo = 0u;
        const float z = znext;
        if (k + 32u < n) // the next step's load while this one is folded in
            znext = b.csr_z[start + k + 32u];
        if (k < n)
        {
            const float f = floorf(2.0f * z);
            if (f >= static_cast<float>(q0) && f < static_cast<float>(q0 + nb))
            {
                q = static_cast<int32_t>(f) - q0;
                zo = zord(z);
            }
            else
                bad = true; // nan or outside the bucket range
        }
        uint32_t todo = __ballot_sync(0xffffffffu, q >= 0);
        while (todo)
        {
            const int32_t lq = __shfl_sync(0xffffffffu, q, __ffs(todo) - 1);
            const bool mine = q == lq;
            const uint32_t gm = __ballot_sync(0xffffffffu, mine);
            const uint32_t glo = __reduce_min_sync(0xffffffffu, mine ? zo : 0xffffffffu);
            const uint32_t ghi = __reduce_max_sync(0xffffffffu, mine ? zo : 0u);
            if (lane == static_cast<uint32_t>(lq))
            {
                cnt += static_cast<uint32_t>(__popc(gm));
                lo = min(lo, glo);
                hi = max(hi, ghi);
            }
            todo &= ~gm;
        }
    }
    if (__any_sync(0xffffffffu, bad))
        return false;
    // lane q = bucket q: position of its first height, previous non-empty bucket
    const uint32_t below = warp_incl_scan(cnt) - cnt;
    int32_t last = (cnt > 0u) ? static_cast<int32_t>(lane) : -1; // inclusive max-scan of non-empty
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int32_t t = __shfl_up_sync(0xffffffffu, last, o);
        if (lane >= static_cast<uint32_t>(o))
            last = max(last, t);
    }
    int32_t prev = __shfl_up_sync(0xffffffffu, last, 1);
    if (lane == 0)
        prev = -1;
    const uint32_t hprev = __shfl_sync(0xffffffffu, hi, max(prev, 0));
    bool qual = false;
    if (cnt > 0u && prev >= 0 && below <= n / 2)
        qual = (zunord(lo) - zunord(hprev)) > 0.5F;
    const uint32_t qm = __ballot_sync(0xffffffffu, qual);
    const uint32_t ne = __ballot_sync(0xffffffffu, cnt > 0u);
    const int32_t pick = qm ? (31 - __clz(qm)) : (__ffs(ne) - 1); // no boundary: z[0], the lowest bucket
    const uint32_t zpick = __shfl_sync(0xffffffffu, lo, pick);
    if (lane == 0)
        b.zlow[c] = zunord(zpick);
    return true;
}

// Fallback for a cell the buckets cannot take (at most kMediumCell heights): warp bitonic sort.
__device__ __forceinline__ void cell_zlow_sorted(const BatchDev& b, uint32_t c, uint32_t n, uint32_t start, float* zs)
{
    const uint32_t lane = lane_id();
    const uint32_t np2 = next_pow2(n);
    for (uint32_t k = lane; k < np2; k += 32)
        zs[k] = (k < n) ? b.csr_z[start + k] : INFINITY;
    __syncwarp();
    warp_bitonic_smem(zs, np2, [](float a, float bb) { return a < bb; });
    int kbest = 0;
    for (uint32_t k = 1 + lane; k <= n / 2; k += 32)
        if (zs[k] - zs[k - 1] > 0.5F)
            kbest = static_cast<int>(k); // lanes visit k in increasing order
    kbest = static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<unsigned>(kbest)));
    if (lane == 0)
        b.zlow[c] = zs[kbest];
    __syncwarp();
}

// One azimuth slice of the polar grid per CTA: the lowest heights of its cells (segmenter.cpp:249-260),
// the RECM elevation chain along it (:215-267) and the RANSAC candidates of its near cells (:345-357:
// points whose height is within 2 thr of the elevation). Bound by latency (a handful of dependent loads
// per cell, then the chain): as six launches (cells, large cells, chain, candidate counts, their
// scan, candidates) the steps took 90 us of a 64 x 2048 scan, four fifths of it launches and tails.
// The candidates keep no order: the inlier counts need none, and the few that the hypotheses draw by
// rank are found by selection in k_ransac_draw. (Ordering every near cell's points for them was most
// of the cells' time.)
constexpr uint32_t kRecmThreads = 256;
constexpr uint32_t kRecmTable = 2048; // buckets of a slice in shared memory (50 cells x 15 by default)

struct RecmSmem
{
    float sz[kLargeCellMax]; // the slice's bucket table, then heights to be sorted
    uint32_t nlarge, nbad, ccount[kRecmThreads / 32], cbase[kRecmThreads / 32];
    int32_t sk;
};

// Slice g of the batch, by a CTA.
__device__ __forceinline__ void recm_slice(const BatchDev& b, uint32_t g, RecmSmem& sh)
{
    static_assert(4u * kRecmTable <= kLargeCellMax, "counts, minima, maxima and the cells' starts");
    static_assert(kRecmThreads / 32 * kMediumCell <= kLargeCellMax, "the warps' parts fit");
    float* sz = sh.sz;
    uint32_t &nlarge = sh.nlarge, &nbad = sh.nbad, *ccount = sh.ccount, *cbase = sh.cbase;
    int32_t& sk = sh.sk;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const int s = scan_of_slice(b, g);
    const ScanDev& sd = b.scans[s];
    const uint32_t slice = g - sd.slice_off;
    const uint32_t off = sd.cell_off + slice * static_cast<uint32_t>(sd.nrad);
    if (threadIdx.x == 0)
        nlarge = nbad = 0u;
    __syncthreads();
    const int32_t q0 = static_cast<int32_t>(floorf(2.0f * sd.zmin_adj));
    const int32_t nb = static_cast<int32_t>(floorf(2.0f * sd.zmax_adj)) - q0 + 1;
    const uint32_t nr = static_cast<uint32_t>(sd.nrad);
    if (nb >= 1 && nb <= 32 && nr * static_cast<uint32_t>(nb) <= kRecmTable)
    {
        // all buckets of the slice's cells in one table (bucket-major): the slice's points, which lie
        // behind one another in the lists, are folded in one per thread, then a thread per cell
        // walks its buckets (see cell_zlow_hist for the rule)
        uint32_t* tcnt = reinterpret_cast<uint32_t*>(sz);
        uint32_t *tlo = tcnt + kRecmTable, *thi = tlo + kRecmTable, *first = thi + kRecmTable;
        for (uint32_t k = threadIdx.x; k < nr * static_cast<uint32_t>(nb); k += kRecmThreads)
        {
            tcnt[k] = 0u;
            tlo[k] = 0xffffffffu;
            thi[k] = 0u;
        }
        for (uint32_t k = threadIdx.x; k < nr; k += kRecmThreads)
            first[k] = b.cell_start[off + k];
        __syncthreads();
        const uint32_t p0 = first[0], p1 = first[nr - 1u] + b.cell_cnt[off + nr - 1u];
        for (uint32_t k = p0 + threadIdx.x; k < p1; k += kRecmThreads)
        {
            const float z = b.csr_z[k];
            uint32_t lo = 0u, hi = nr - 1u; // the last cell that starts at or before the point
            while (lo < hi)
            {
                const uint32_t mid = (lo + hi + 1u) / 2u;
                if (first[mid] <= k)
                    lo = mid;
                else
                    hi = mid - 1u;
            }
            const float f = floorf(2.0f * z);
            if (f >= static_cast<float>(q0) && f < static_cast<float>(q0 + nb))
            {
                const uint32_t at = static_cast<uint32_t>(static_cast<int32_t>(f) - q0) * nr + lo, zo = zord(z);
                atomicAdd(&tcnt[at], 1u);
                atomicMin(&tlo[at], zo);
                atomicMax(&thi[at], zo);
            }
            // (a nan enters no bucket: its cell's counts stay below the cell's size)
        }
        __syncthreads();
        for (uint32_t c = threadIdx.x; c < nr; c += kRecmThreads)
        {
            const uint32_t n = b.cell_cnt[off + c];
            if (n == 0u)
                continue;
            uint32_t below = 0u, pick = 0u, hprev = 0u;
            bool any = false;
            for (int32_t q = 0; q < nb; ++q)
            {
                const uint32_t at = static_cast<uint32_t>(q) * nr + c, m = tcnt[at];
                if (m == 0u)
                    continue;
                const uint32_t lo = tlo[at];
                if (!any || (below <= n / 2u && (zunord(lo) - zunord(hprev)) > 0.5F))
                    pick = lo; // the lowest bucket, or the last gap in the lower half
                any = true;
                hprev = thi[at];
                below += m;
            }
            b.zlow[off + c] = zunord(pick);
            if (below != n)
                b.large_list[off + atomicAdd(&nbad, 1u)] = off + c;
        }
        __syncthreads();
        // cells with a nan: small ones sorted by a warp, the others stay listed (behind a counter of their own: the
        // other warps only meet this one at the barrier below)
        if (warp == 0)
            for (uint32_t li = 0; li < nbad; ++li)
            {
                const uint32_t c = b.large_list[off + li], n = b.cell_cnt[c];
                __syncwarp();
                if (n <= static_cast<uint32_t>(kMediumCell))
                    cell_zlow_sorted(b, c, n, b.cell_start[c], sz);
                else if (lane == 0)
                    b.large_list[off + nlarge++] = c; // nlarge <= li
                __syncwarp();
            }
    }
    else
    {
        // more buckets than the table holds: every eighth occupied cell per warp
        uint32_t turn = 0u;
        for (int32_t r0 = 0; r0 < sd.nrad; r0 += 32)
        {
            const int32_t r = r0 + static_cast<int32_t>(lane);
            const uint32_t cnt = (r < sd.nrad) ? b.cell_cnt[off + static_cast<uint32_t>(r)] : 0u;
            const uint32_t st = (cnt != 0u) ? b.cell_start[off + static_cast<uint32_t>(r)] : 0u;
            for (uint32_t m = __ballot_sync(0xffffffffu, cnt != 0u); m != 0u; m &= m - 1u, ++turn)
            {
                if (turn % (kRecmThreads / 32u) != warp)
                    continue;
                const int j = __ffs(m) - 1;
                const uint32_t c = off + static_cast<uint32_t>(r0 + j);
                const uint32_t n = __shfl_sync(0xffffffffu, cnt, j), start = __shfl_sync(0xffffffffu, st, j);
                if (cell_zlow_hist(b, sd, c, n, start))
                    continue;
                if (n <= static_cast<uint32_t>(kMediumCell))
                    cell_zlow_sorted(b, c, n, start, sz + warp * kMediumCell);
                else if (lane == 0)
                    b.large_list[off + atomicAdd(&nlarge, 1u)] = c; // heights the buckets cannot take: sorted below
            }
        }
    }
    __syncthreads();
    const uint32_t nl = nlarge;
    for (uint32_t li = 0; li < nl; ++li)
    {
        const uint32_t c = b.large_list[off + li];
        const uint32_t n = b.cell_cnt[c], start = b.cell_start[c];
        if (n > kLargeCellMax)
        {
            if (threadIdx.x == 0)
            {
                raise_err(&b.state[s], ERR_CELL_TOO_LARGE);
                b.zlow[c] = b.csr_z[start];
            }
            continue;
        }
        const uint32_t np2 = next_pow2(n);
        for (uint32_t k = threadIdx.x; k < np2; k += blockDim.x)
            sz[k] = (k < n) ? b.csr_z[start + k] : INFINITY;
        if (threadIdx.x == 0)
            sk = 0;
        __syncthreads();
        block_bitonic_sort(sz, np2, [](float x, float y) { return x < y; });
        for (uint32_t k = 1 + threadIdx.x; k <= n / 2; k += blockDim.x)
            if (sz[k] - sz[k - 1] > 0.5F)
                atomicMax(&sk, static_cast<int32_t>(k));
        __syncthreads();
        if (threadIdx.x == 0)
            b.zlow[c] = sz[sk];
        __syncthreads();
    }
    __syncthreads();
    auto link = [&](float prev, uint32_t cnt, float zlo) {
        const float lim = prev + sd.delta;
        return (cnt == 0u) ? lim : ((lim < zlo) ? lim : zlo); // std::min(curr_z_min, prev + delta)
    };
    // the near cells, two warps each: their elevation (at most three links), the candidates counted
    const int32_t rad = static_cast<int32_t>(warp / 2u);
    const uint32_t nc = off + static_cast<uint32_t>(rad);
    float e = -sd.sensor_h + sd.thr;
    for (int32_t r = 1; r <= rad; ++r)
        e = link(e, b.cell_cnt[off + static_cast<uint32_t>(r)], b.zlow[off + static_cast<uint32_t>(r)]);
    const uint32_t n = b.cell_cnt[nc], start = b.cell_start[nc];
    if (n > kLargeCellMax && threadIdx.x % 64u == 0u)
        raise_err(&b.state[s], ERR_CELL_TOO_LARGE); // the capacity of a near cell
    const uint32_t half = ((n + 63u) / 64u) * 32u; // this warp's entries: [i0, i1)
    const uint32_t i0 = (warp & 1u) ? min(half, n) : 0u, i1 = (warp & 1u) ? n : min(half, n);
    const float lim = 2.0F * sd.thr;
    uint32_t found = 0u;
#pragma unroll 4
    for (uint32_t k = i0 + lane; k < i1; k += 32u)
        found += (fabsf(e - b.csr_z[start + k]) < lim) ? 1u : 0u;
    found = warp_sum(found);
    if (lane == 0)
        ccount[warp] = found;
    __syncthreads();
    if (warp == 0)
    {
        // room for the slice's candidates, and the counts per near cell
        const uint32_t v = (lane < kRecmThreads / 32u) ? ccount[lane] : 0u;
        const uint32_t incl = warp_incl_scan(v);
        uint32_t base = 0u;
        if (lane == 31u && incl)
            base = atomicAdd(&b.state[s].n_cand, incl);
        base = __shfl_sync(0xffffffffu, base, 31);
        if (lane < kRecmThreads / 32u)
            cbase[lane] = sd.pt_off + base + incl - v;
        const uint32_t pair = v + __shfl_down_sync(0xffffffffu, v, 1);
        if (lane < kRecmThreads / 32u && (lane & 1u) == 0u)
            b.near_cnt[sd.near_off + slice * static_cast<uint32_t>(kRansacRadialBins) + lane / 2u] = pair;
    }
    __syncthreads();
    uint32_t pos = cbase[warp];
    for (uint32_t k0 = i0; k0 < i1; k0 += 32u)
    {
        const uint32_t k = k0 + lane;
        const bool pred = k < i1 && fabsf(e - b.csr_z[start + k]) < lim;
        const uint32_t m = __ballot_sync(0xffffffffu, pred);
        if (pred)
        {
            const float4 p = b.pts[sd.pt_off + static_cast<uint32_t>(b.csr_idx[start + k])];
            b.cand[pos + static_cast<uint32_t>(__popc(m & ((1u << lane) - 1u)))] = make_float4(p.x, p.y, p.z, 0.0f);
        }
        pos += static_cast<uint32_t>(__popc(m));
    }
    // the chain along the whole slice (the last warp: its near cell is the sparsest), 32 cells at a time
    if (warp != kRecmThreads / 32u - 1u)
        return;
    float prev = -sd.sensor_h + sd.thr;
    for (int32_t r0 = 0; r0 < sd.nrad; r0 += 32)
    {
        const int32_t r = r0 + static_cast<int32_t>(lane);
        const uint32_t cnt = (r < sd.nrad) ? b.cell_cnt[off + static_cast<uint32_t>(r)] : 0u;
        const float zlo = (r < sd.nrad && cnt != 0u) ? b.zlow[off + static_cast<uint32_t>(r)] : 0.0f;
        float mine = prev;
#pragma unroll 8
        for (int j = 0; j < 32; ++j)
        {
            const uint32_t cj = __shfl_sync(0xffffffffu, cnt, j);
            const float zj = __shfl_sync(0xffffffffu, zlo, j);
            if (r0 + j > 0)
                prev = link(prev, cj, zj);
            if (static_cast<int>(lane) == j)
                mine = prev;
        }
        if (r < sd.nrad)
            b.elev[off + static_cast<uint32_t>(r)] = mine;
    }
}

__global__ void __launch_bounds__(kRecmThreads) k_recm(BatchDev b)
{
    pdl_enter();
    __shared__ RecmSmem sh;
    recm_slice(b, blockIdx.x, sh);
}

// Slice g by a warp, a point per lane: false, with nothing written, where it holds more than 32 or a NaN height.
// Elevations only where a point lies (nothing reads the others).
__device__ __forceinline__ bool recm_slice_few(const BatchDev& b, uint32_t g)
{
    const uint32_t lane = lane_id();
    const int s = scan_of_slice(b, g);
    const ScanDev& sd = b.scans[s];
    const uint32_t slice = g - sd.slice_off;
    const uint32_t off = sd.cell_off + slice * static_cast<uint32_t>(sd.nrad);
    const uint32_t p0 = b.cell_start[off], n = b.cell_start[off + static_cast<uint32_t>(sd.nrad)] - p0;
    if (n > 32u)
        return false;
    const bool in = lane < n;
    const uint32_t at = in ? sd.pt_off + static_cast<uint32_t>(b.csr_idx[p0 + lane]) : 0u;
    const float z = in ? b.csr_z[p0 + lane] : 0.0f;
    const uint32_t r = in ? static_cast<uint32_t>(b.pt_cell[at]) - off : 0xffffffffu;
    if (__any_sync(0xffffffffu, z != z))
        return false;
    // the point's place among its cell's heights, the one below it, the cell's size (see cell_zlow_hist for the rule)
    uint32_t rank = 0u, size = 0u;
    float below = -INFINITY;
    for (uint32_t j = 0; j < n; ++j)
    {
        const float zj = __shfl_sync(0xffffffffu, z, static_cast<int>(j));
        const bool mate = __shfl_sync(0xffffffffu, r, static_cast<int>(j)) == r;
        const bool before = mate && (zj < z || (zj == z && j < lane));
        size += mate ? 1u : 0u;
        rank += before ? 1u : 0u;
        below = before ? fmaxf(below, zj) : below;
    }
    const bool gap = rank >= 1u && rank <= size / 2u && (z - below) > 0.5F;
    // the chain along the slice, occupied cell by occupied cell
    float e = -sd.sensor_h + sd.thr, mine = e;
    bool open = in;
    for (uint32_t last = 0u;;)
    {
        const uint32_t next = __reduce_min_sync(0xffffffffu, open ? r : 0xffffffffu);
        if (next == 0xffffffffu)
            break;
        for (; last + 1u < next; ++last)
            e = e + sd.delta;
        const bool member = open && r == next;
        const uint32_t key = !member ? 0u : (gap ? rank + 1u : (rank == 0u ? 1u : 0u)); // the last gap, or the lowest
        const uint32_t best = __reduce_max_sync(0xffffffffu, key);
        const int src = __ffs(__ballot_sync(0xffffffffu, member && key == best)) - 1;
        const float zlo = __shfl_sync(0xffffffffu, z, src);
        if (next != 0u)
        {
            const float lim = e + sd.delta;
            e = (lim < zlo) ? lim : zlo;
        }
        if (static_cast<int>(lane) == src)
            b.elev[off + next] = e;
        mine = member ? e : mine;
        open = open && !member;
        last = next;
    }
    // the candidates of the near cells
    const bool cand = in && r < static_cast<uint32_t>(kRansacRadialBins) && fabsf(mine - z) < 2.0F * sd.thr;
    const uint32_t all = __ballot_sync(0xffffffffu, cand);
    uint32_t count = 0u, base = 0u;
#pragma unroll
    for (uint32_t q = 0; q < static_cast<uint32_t>(kRansacRadialBins); ++q)
    {
        const uint32_t m = __ballot_sync(0xffffffffu, cand && r == q);
        count = (lane == q) ? static_cast<uint32_t>(__popc(m)) : count;
    }
    if (lane < static_cast<uint32_t>(kRansacRadialBins))
        b.near_cnt[sd.near_off + slice * static_cast<uint32_t>(kRansacRadialBins) + lane] = count;
    if (lane == 0u && all)
        base = atomicAdd(&b.state[s].n_cand, static_cast<uint32_t>(__popc(all)));
    base = sd.pt_off + __shfl_sync(0xffffffffu, base, 0);
    if (cand)
    {
        const float4 p = b.pts[at];
        b.cand[base + static_cast<uint32_t>(__popc(all & ((1u << lane) - 1u)))] = make_float4(p.x, p.y, p.z, 0.0f);
    }
    return true;
}

// Batches of few points a slice: eight slices per CTA, a warp for each that holds few, the others by the CTA one after the
// other. A CTA per slice holds an SM's shared memory for 6 us whatever it holds: 1,000 scans of 300 points took 2.2 ms,
// 4,000 of them 9.2 (the six kernels before k_recm about half of it), now 0.24 and 0.8. Below 16 points a slice on average:
// most hold up to 32 then (256 scans of 3,000 points, 8 a slice: 0.68 -> 0.15 ms).
__global__ void __launch_bounds__(kRecmThreads) k_recm_sparse(BatchDev b, uint32_t nslices)
{
    pdl_enter();
    __shared__ RecmSmem sh;
    __shared__ uint32_t rest;
    const uint32_t first = blockIdx.x * (kRecmThreads / 32u), warp = threadIdx.x >> 5;
    if (threadIdx.x == 0)
        rest = 0u;
    __syncthreads();
    if (first + warp < nslices && !recm_slice_few(b, first + warp) && lane_id() == 0u)
        atomicOr(&rest, 1u << warp);
    __syncthreads();
    for (uint32_t m = rest; m != 0u; m &= m - 1u)
    {
        recm_slice(b, first + static_cast<uint32_t>(__ffs(m) - 1), sh);
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// RANSAC near-field correction (correctCloseRangeFalsePositivesRANSAC, segmenter.cpp:321-479).
// ------------------------------------------------------------------------------------------
// MT19937 (Matsumoto & Nishimura, 1998) and Lemire's nearly divisionless bounded draw
// (Lemire, "Fast Random Integer Generation in an Interval", 2019), which is how
// std::uniform_int_distribution<uint32_t> maps a 32-bit engine onto [0, n-1].
struct Mt19937
{
    uint32_t mt[624];
    int idx;
    __device__ void seed(uint32_t s)
    {
        mt[0] = s;
        for (int i = 1; i < 624; ++i)
            mt[i] = 1812433253u * (mt[i - 1] ^ (mt[i - 1] >> 30)) + static_cast<uint32_t>(i);
        idx = 624;
    }
    __device__ void twist()
    {
        for (int i = 0; i < 624; ++i)
        {
            const uint32_t y = (mt[i] & 0x80000000u) | (mt[(i + 1) % 624] & 0x7fffffffu);
            mt[i] = mt[(i + 397) % 624] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
        }
        idx = 0;
    }
    __device__ uint32_t next()
    {
        if (idx >= 624)
            twist();
        uint32_t y = mt[idx++];
        y ^= y >> 11;
        y ^= (y << 7) & 0x9d2c5680u;
        y ^= (y << 15) & 0xefc60000u;
        y ^= y >> 18;
        return y;
    }
};

// Every scan draws from MT19937 seeded with 42 (segmenter.cpp:328), so its first outputs are the
// same for all scans: they are computed once per device on the host (std::mt19937) and read from
// this table; a scan that needs more (many redraws) runs the generator itself past the table.
constexpr int kMtTable = 4 * 624;
static_assert(kMtTable % 4 == 0, "copied as 16-byte words");
__device__ __align__(16) uint32_t g_mt42[kMtTable];

struct Mt42Stream
{
    const uint32_t* table; // the first kMtTable outputs (a shared-memory copy of g_mt42)
    Mt19937 gen;           // seeded only past the table
    int idx = 0;
    __device__ uint32_t next()
    {
        if (idx < kMtTable)
            return table[idx++];
        if (idx == kMtTable)
        {
            gen.seed(42u);
            for (int k = 0; k < kMtTable; ++k)
                gen.next();
        }
        ++idx;
        return gen.next();
    }
    __device__ uint32_t bounded(uint32_t range) // uniform in [0, range)
    {
        uint64_t m = static_cast<uint64_t>(next()) * range;
        uint32_t l = static_cast<uint32_t>(m);
        if (l < range)
        {
            const uint32_t t = (0u - range) % range;
            while (l < t)
            {
                m = static_cast<uint64_t>(next()) * range;
                l = static_cast<uint32_t>(m);
            }
        }
        return static_cast<uint32_t>(m >> 32);
    }
};

// The r-th smallest index among a near cell's candidates (entries [start, start + n) of the polar
// grid's lists, those within `lim` of elevation e; indices below `end`), by one warp. While more than
// kSelect entries are in question, a pass counts them in 32 equal index ranges and keeps the one that
// holds the rank; the rest is gathered once and bisected in registers (a pass over memory costs far
// more than the 17 or so steps).
constexpr uint32_t kSelect = 256;

__device__ __forceinline__ uint32_t select_candidate(const BatchDev& b, uint32_t start, uint32_t n, float e, float lim,
                                                     uint32_t r, uint32_t end, uint32_t* buf)
{
    const uint32_t lane = lane_id();
    uint32_t lo = 0u, active = n; // indices in [lo, end)
    while (active > kSelect && end - lo > 1u)
    {
        const uint32_t width = (end - lo + 31u) / 32u;
        buf[lane] = 0u;
        __syncwarp();
#pragma unroll 4
        for (uint32_t k = lane; k < n; k += 32u)
        {
            const uint32_t v = static_cast<uint32_t>(b.csr_idx[start + k]);
            if (v >= lo && v < end && fabsf(e - b.csr_z[start + k]) < lim)
                atomicAdd(&buf[(v - lo) / width], 1u);
        }
        __syncwarp();
        const uint32_t c = buf[lane];
        const uint32_t incl = warp_incl_scan(c);
        const uint32_t pick = static_cast<uint32_t>(__ffs(__ballot_sync(0xffffffffu, incl > r)) - 1) & 31u; // r < candidates
        r -= __shfl_sync(0xffffffffu, incl - c, static_cast<int>(pick));
        active = __shfl_sync(0xffffffffu, c, static_cast<int>(pick));
        lo += pick * width;
        end = min(end, lo + width);
        __syncwarp();
    }
    uint32_t m = 0u;
#pragma unroll 4
    for (uint32_t k0 = 0; k0 < n; k0 += 32u)
    {
        const uint32_t k = k0 + lane;
        const uint32_t v = (k < n) ? static_cast<uint32_t>(b.csr_idx[start + k]) : 0u;
        const bool in = k < n && v >= lo && v < end && fabsf(e - b.csr_z[start + k]) < lim;
        const uint32_t mask = __ballot_sync(0xffffffffu, in);
        const uint32_t at = m + static_cast<uint32_t>(__popc(mask & ((1u << lane) - 1u)));
        if (in && at < kSelect)
            buf[at] = v;
        m += static_cast<uint32_t>(__popc(mask));
    }
    __syncwarp();
    m = min(m, kSelect);
    uint32_t v[kSelect / 32u];
#pragma unroll
    for (uint32_t q = 0; q < kSelect / 32u; ++q)
        v[q] = (q * 32u + lane < m) ? buf[q * 32u + lane] : 0xffffffffu;
    uint32_t x = lo; // the smallest value with more than r entries up to it
    for (uint32_t step = (end - lo > 1u) ? 1u << (31 - __clz(static_cast<int>(end - lo - 1u))) : 0u; step != 0u; step >>= 1)
    {
        uint32_t below = 0u; // entries below x + step
#pragma unroll
        for (uint32_t q = 0; q < kSelect / 32u; ++q)
            if (q * 32u < m)
                below += static_cast<uint32_t>(__popc(__ballot_sync(0xffffffffu, v[q] < x + step)));
        if (below <= r)
            x += step;
    }
    __syncwarp();
    return x;
}

// The hypotheses' points and planes (segmenter.cpp:359-407), kDrawCtas CTAs per scan, each for its share
// of the hypotheses. The draws index the candidates in (slice, radial bin, cloud) order: the near cell
// comes from the scan of the cells' candidate counts, the point by selection within the cell.
// Hypothesis it takes outputs 2 it and 2 it + 1 of the seed-42 stream unless an earlier draw was
// rejected or repeated (a rejected draw shifts every later one): all draws are checked at once, and only
// then one thread walks the stream. With lane 0 walking it always, and ordered candidates, 20 us.
constexpr uint32_t kDrawThreads = 1024; // a warp per draw
constexpr uint32_t kDrawCtas = kNearCopies;
constexpr uint32_t kDrawPer = (kMaxRansacIters + kDrawCtas - 1) / kDrawCtas; // hypotheses per CTA

__global__ void __launch_bounds__(kDrawThreads) k_ransac_draw(BatchDev b)
{
    pdl_enter();
    __shared__ uint32_t di[2 * kMaxRansacIters]; // i2, i3 of every hypothesis
    __shared__ float4 pt[2 * kDrawPer];
    __shared__ uint32_t sel[kDrawThreads / 32][kSelect];
    __shared__ uint32_t sm[33];
    __shared__ int bad;
    const int s = static_cast<int>(blockIdx.x / kDrawCtas);
    const uint32_t part = blockIdx.x % kDrawCtas;
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const ScanDev& sd = b.scans[s];
    ScanState& st = b.state[s];
    const uint32_t N = st.n_cand;
    if (part == 0u && tid == 0)
        st.cand_off = sd.pt_off;
    if (N < 2)
        return; // the reference never ends its p3 draw for N == 1 (segmenter.cpp:382-386)
    // near cells: first candidate rank of each (this CTA's copy)
    const uint32_t cells = static_cast<uint32_t>(sd.nslice * sd.nnear_per_slice);
    uint32_t* rank = b.near_start + static_cast<size_t>(part) * b.nnear + sd.near_off;
    uint32_t base = 0u;
    for (uint32_t k0 = 0; k0 < cells; k0 += kDrawThreads)
    {
        const uint32_t k = k0 + tid;
        const uint32_t v = (k < cells) ? b.near_cnt[sd.near_off + k] : 0u;
        uint32_t total;
        const uint32_t at = base + block_excl_scan(v, sm, &total);
        if (k < cells)
            rank[k] = at;
        base += total;
    }
    // the draws as if none were rejected or repeated
    bool odd = false;
    if (tid < 2u * kMaxRansacIters)
    {
        const uint64_t m = static_cast<uint64_t>(g_mt42[tid]) * N;
        const uint32_t l = static_cast<uint32_t>(m);
        odd = l < N && l < (0u - N) % N;
        di[tid] = static_cast<uint32_t>(m >> 32);
    }
    if (tid == 0)
        bad = 0;
    __syncthreads();
    odd |= tid < static_cast<uint32_t>(kMaxRansacIters) && di[2u * tid] == di[2u * tid + 1u];
    if (__syncthreads_or(odd))
    {
        if (tid == 0)
        {
            Mt42Stream gen;
            gen.table = g_mt42;
            for (int it = 0; it < kMaxRansacIters; ++it)
            {
                const uint32_t i2 = gen.bounded(N);
                uint32_t i3 = gen.bounded(N);
                int guard = 0;
                while (i3 == i2 && guard < (1 << 20))
                {
                    i3 = gen.bounded(N);
                    ++guard;
                }
                if (guard >= (1 << 20))
                {
                    bad = 1;
                    break;
                }
                di[2 * it] = i2;
                di[2 * it + 1] = i3;
            }
        }
        __syncthreads();
        if (bad)
        {
            if (part == 0u && tid == 0)
                raise_err(&st, ERR_INTERNAL);
            return;
        }
    }
    const uint32_t it0 = part * kDrawPer, it1 = min(it0 + kDrawPer, static_cast<uint32_t>(kMaxRansacIters));
    const float lim = 2.0F * sd.thr;
    for (uint32_t d = warp; d < 2u * (it1 - it0); d += kDrawThreads / 32u)
    {
        const uint32_t i = di[2u * it0 + d];
        uint32_t lo = 0u; // the last cell whose first rank is not above i, 32 probes a step
        for (uint32_t len = cells; len > 1u;)
        {
            const uint32_t w = (len + 31u) / 32u;
            const bool at = lane * w < len && rank[lo + lane * w] <= i; // (true for lane 0)
            const uint32_t k = static_cast<uint32_t>(__popc(__ballot_sync(0xffffffffu, at))) - 1u;
            lo += k * w;
            len = min(w, len - k * w);
        }
        const uint32_t c = sd.cell_off + (lo / static_cast<uint32_t>(sd.nnear_per_slice)) * static_cast<uint32_t>(sd.nrad) +
                           lo % static_cast<uint32_t>(sd.nnear_per_slice);
        const uint32_t idx = select_candidate(b, b.cell_start[c], b.cell_cnt[c], b.elev[c], lim, i - rank[lo], st.n_pts, sel[warp]);
        if (lane == 0)
            pt[d] = b.pts[sd.pt_off + min(idx, sd.n - 1u)];
    }
    __syncthreads();
    const uint32_t it = it0 + tid;
    bool ok = false;
    if (it < it1)
    {
        const float p1x = 0.0F, p1y = 0.0F, p1z = -sd.sensor_h;
        const float4 p2 = pt[2u * tid], p3 = pt[2u * tid + 1u];
        float nx = ((p2.y - p1y) * (p3.z - p1z)) - ((p2.z - p1z) * (p3.y - p1y));
        float ny = ((p2.z - p1z) * (p3.x - p1x)) - ((p2.x - p1x) * (p3.z - p1z));
        float nz = ((p2.x - p1x) * (p3.y - p1y)) - ((p2.y - p1y) * (p3.x - p1x));
        const float den = (nx * nx) + (ny * ny) + (nz * nz);
        float4 pl = make_float4(0, 0, 0, 0);
        if (!(den < 1.0e-5F))
        {
            const float norm = 1.0F / sqrtf(den);
            nz *= norm;
            if (!(fabsf(nz) < sd.max_cos))
            {
                nx *= norm;
                ny *= norm;
                const float pd = (nx * p1x) + (ny * p1y) + (nz * p1z);
                pl = make_float4(nx, ny, nz, pd);
                ok = true;
            }
        }
        b.planes[s * kMaxRansacIters + static_cast<int>(it)] = pl;
    }
    static_assert(kDrawPer <= 32u, "one warp fits the CTA's planes");
    const unsigned long long valid = static_cast<unsigned long long>(__ballot_sync(0xffffffffu, ok)) << it0;
    if (tid == 0 && valid)
        atomicOr(&b.pvalid[s], valid);
}

// Inlier counts of every hypothesis plane of a scan (segmenter.cpp:409-430): lane l of every
// warp holds planes l and l + 32 as a float pair and counts, for the candidates its warp takes,
// |((n.x p.x + n.y p.y) + n.z p.z) - d| < thr with packed binary32 operations (each half rounds
// like the scalar operation, in the reference's order). The work is a flat list of tiles of
// kTile candidates over the batch's scans with usable planes (scan by scan, so a tile
// belongs to one scan), taken grid-strided: a large scan spreads over the whole grid instead of
// its own share of it. A CTA's tiles come in increasing order, so it follows the scans with a
// cursor, loads a scan's planes when it reaches it and adds its counts when it leaves it (integer
// partial counts add up exactly). The last CTA to finish picks every scan's plane (segmenter.cpp:432-443).
// Batches whose points do not give every CTA a tile of 1,024 take tiles of 256: a warp's 128 candidates in a row
// were most of the time (32 x 1024 scan 15 -> 9 us, 64 x 2048 16 -> 11, 128 x 4096 19 -> 13).
constexpr uint32_t kInlierTile = 1024;
constexpr uint32_t kInlierTileFew = 256;

__device__ __forceinline__ void ransac_select(const BatchDev& b, int s)
{
    ScanState& st = b.state[s];
    const unsigned long long valid = b.pvalid[s];
    // a warp: the first hypothesis of the most inliers, two per lane
    const uint32_t lane = lane_id();
    auto count = [&](uint32_t it) {
        return it < static_cast<uint32_t>(kMaxRansacIters) && ((valid >> it) & 1ull) ? __ldcg(&b.inliers[s * kMaxRansacIters + it]) : 0u;
    };
    const uint32_t n0 = count(lane), n1 = count(lane + 32u);
    const uint32_t best = __reduce_max_sync(0xffffffffu, max(n0, n1));
    const uint32_t m0 = __ballot_sync(0xffffffffu, n0 == best), m1 = __ballot_sync(0xffffffffu, n1 == best);
    const int bi = m0 ? __ffs(m0) - 1 : 31 + __ffs(m1);
    if (lane != 0u)
        return;
    if (best > 0)
    {
        float4 q = b.planes[s * kMaxRansacIters + bi];
        if (q.z < 0)
        {
            q.x = -q.x;
            q.y = -q.y;
            q.z = -q.z;
            q.w = -q.w;
        }
        st.plane[0] = q.x;
        st.plane[1] = q.y;
        st.plane[2] = q.z;
        st.plane[3] = q.w;
        st.ransac_ok = 1;
    }
}

template <uint32_t kTile>
__global__ void __launch_bounds__(256) k_ransac_inliers(BatchDev b)
{
    pdl_enter();
    static_assert(kMaxRansacIters <= 64, "two planes per lane");
    __shared__ float4 tile[kTile];
    const uint32_t lane = lane_id();
    const uint32_t i0 = lane, i1 = lane + 32u;
    const uint32_t warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto tiles_of = [&](int q) -> uint32_t {
        return (b.pvalid[q] != 0ull) ? div_up(b.state[q].n_cand, kTile) : 0u;
    };
    int cs = 0; // the cursor: scan cs owns tiles [cbase, cbase + ctiles)
    uint32_t cbase = 0u, ctiles = (b.nscan > 0) ? tiles_of(0) : 0u;
    int s = -1; // the scan whose planes are loaded
    unsigned long long valid = 0ull;
    float2 qx = make_float2(0.f, 0.f), qy = qx, qz = qx, nqw = qx;
    float thr = 0.0f;
    uint32_t ca = 0u, cb = 0u;
    // The planes' counters take one atomic at a time. With small tiles (few points, many CTAs for them) a CTA's warps
    // add up in shared memory first; with large ones a CTA meets several scans, and the barriers cost more.
    constexpr bool together = kTile < kInlierTile;
    __shared__ uint32_t sum[together ? 64 : 1];
    if (together)
    {
        if (threadIdx.x < 64u)
            sum[threadIdx.x] = 0u;
        __syncthreads();
    }
    auto flush = [&]() { // (all threads alike)
        if (s < 0)
            return;
        if constexpr (!together)
        {
            if (i0 < static_cast<uint32_t>(kMaxRansacIters) && ((valid >> i0) & 1ull) && ca)
                atomicAdd(&b.inliers[s * kMaxRansacIters + i0], ca);
            if (i1 < static_cast<uint32_t>(kMaxRansacIters) && ((valid >> i1) & 1ull) && cb)
                atomicAdd(&b.inliers[s * kMaxRansacIters + i1], cb);
            ca = cb = 0u;
        }
        else
        {
            if (ca)
                atomicAdd(&sum[i0], ca);
            if (cb)
                atomicAdd(&sum[i1], cb);
            ca = cb = 0u;
            __syncthreads();
            if (threadIdx.x < 64u)
            {
                const uint32_t n = sum[threadIdx.x];
                sum[threadIdx.x] = 0u;
                if (n && threadIdx.x < static_cast<uint32_t>(kMaxRansacIters) && ((valid >> threadIdx.x) & 1ull))
                    atomicAdd(&b.inliers[s * kMaxRansacIters + threadIdx.x], n);
            }
            __syncthreads();
        }
    };
    for (uint32_t it = blockIdx.x;; it += gridDim.x)
    {
        while (cs < b.nscan && it >= cbase + ctiles)
        {
            cbase += ctiles;
            ++cs;
            ctiles = (cs < b.nscan) ? tiles_of(cs) : 0u;
        }
        if (cs >= b.nscan)
            break; // uniform over the block
        if (cs != s)
        {
            flush();
            s = cs;
            valid = b.pvalid[s];
            const float4 qa = (i0 < static_cast<uint32_t>(kMaxRansacIters)) ? b.planes[s * kMaxRansacIters + i0] : zero;
            const float4 qb = (i1 < static_cast<uint32_t>(kMaxRansacIters)) ? b.planes[s * kMaxRansacIters + i1] : zero;
            qx = make_float2(qa.x, qb.x);
            qy = make_float2(qa.y, qb.y);
            qz = make_float2(qa.z, qb.z);
            nqw = make_float2(-qa.w, -qb.w); // x - w == x + (-w) exactly
            thr = b.scans[s].thr;
        }
        const ScanState& st = b.state[s];
        const uint32_t base = (it - cbase) * kTile;
        const uint32_t cnt = min(kTile, st.n_cand - base);
        const float4* cand = b.cand + st.cand_off + base;
        // candidates staged in shared memory (coalesced), read by each warp as broadcasts
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x)
            tile[k] = cand[k];
        __syncthreads();
#pragma unroll 4
        for (uint32_t k = warp; k < cnt; k += nwarp)
        {
            const float4 p = tile[k];
            float2 t = __fmul2_rn(qx, make_float2(p.x, p.x));
            t = __fadd2_rn(t, __fmul2_rn(qy, make_float2(p.y, p.y)));
            t = __fadd2_rn(t, __fmul2_rn(qz, make_float2(p.z, p.z)));
            t = __fadd2_rn(t, nqw);
            ca += (fabsf(t.x) < thr) ? 1u : 0u;
            cb += (fabsf(t.y) < thr) ? 1u : 0u;
        }
    }
    flush();
    __shared__ bool last;
    __threadfence(); // this CTA's counts before its ticket
    __syncthreads();
    if (threadIdx.x == 0)
        last = atomicAdd(b.ransac_done, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!last)
        return;
    __threadfence();
    for (int q = static_cast<int>(warp); q < b.nscan; q += static_cast<int>(nwarp))
        ransac_select(b, q);
}

// ------------------------------------------------------------------------------------------
// Labels and range-image projection (segmenter.cpp:269-318 + the RANSAC relabel :445-478).
// Per pixel the winner is the lexicographic minimum of (x^2+y^2, cell, cloud index), the
// order in which the reference's strict '<' visits candidates.
// ------------------------------------------------------------------------------------------
// kPacked: the whole choice in one atomic, point of the least (distance, cell, index) with its label in the last bit, so
// that neither the second pass (k_project_key) nor a look-up of the chosen point's label is needed. Where a scan's
// distances, cells and points need more than 63 bits (e.g. from no least distance on and more than 2^17
// points of a 2 degree grid), two passes: the least distance first. 64 scans: 54 + 58 + 72 us with
// k_project_key and k_pixel in two passes, 60 + 66 us in one.
template <bool kPacked>
__global__ void k_label_depth(BatchDev b)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.npts)
        return;
    const int32_t c = b.pt_cell[i];
    const float4 p = b.pts[i];
    const int32_t pix = b.pt_pix[i];
    if (c < 0)
        return;
    const int s = scan_of_point(b, i);
    const ScanDev& sd = b.scans[s];
    const ScanState& st = b.state[s];
    uint8_t lbl = (p.z >= b.elev[c] + sd.thr) ? LP_LABEL_OBSTACLE : LP_LABEL_GROUND;
    const int32_t radial = static_cast<int32_t>((static_cast<uint32_t>(c) - sd.cell_off) % static_cast<uint32_t>(sd.nrad));
    if (radial < kRansacRadialBins && st.ransac_ok)
    {
        const float sdist = (st.plane[0] * p.x) + (st.plane[1] * p.y) + (st.plane[2] * p.z) - st.plane[3];
        if (sdist < sd.thr)
            lbl = LP_LABEL_GROUND;
    }
    const float d2 = (p.x * p.x) + (p.y * p.y);
    if (kPacked)
    {
        const unsigned long long key =
            // (a nan lies beyond every distance)
            (min(static_cast<unsigned long long>(__float_as_uint(d2) - sd.key_base), (1ull << (63u - sd.key_dist)) - 1ull)
             << sd.key_dist) |
            (static_cast<unsigned long long>(static_cast<uint32_t>(c) - sd.cell_off) << sd.key_cell) |
            (static_cast<unsigned long long>(i - sd.pt_off) << 1) | (lbl == LP_LABEL_GROUND ? 0u : 1u);
        atomicMin(&b.pix_key[sd.pix_off + static_cast<uint32_t>(pix)], key);
        return;
    }
    b.pt_label[i] = lbl;
    atomicMin(&b.pix_depth[sd.pix_off + static_cast<uint32_t>(pix)], __float_as_uint(d2));
}

__global__ void k_project_key(BatchDev b)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.npts)
        return;
    const int32_t c = b.pt_cell[i];
    const float4 p = b.pts[i];
    const int32_t lpix = b.pt_pix[i];
    if (c < 0)
        return;
    const int s = scan_of_point(b, i);
    const ScanDev& sd = b.scans[s];
    const float d2 = (p.x * p.x) + (p.y * p.y);
    const uint32_t pix = sd.pix_off + static_cast<uint32_t>(lpix);
    if (__float_as_uint(d2) != b.pix_depth[pix])
        return;
    const unsigned long long key = (static_cast<unsigned long long>(static_cast<uint32_t>(c) - sd.cell_off) << 32) |
                                   static_cast<unsigned long long>(i - sd.pt_off);
    atomicMin(&b.pix_key[pix], key);
}

// kPer pixels per thread: four (16-byte loads and stores) where they fill the SMs (64 scans: 66 us with one, 39 with
// four), one where they do not.
template <bool kPacked, uint32_t kPer>
__global__ void k_pixel(BatchDev b)
{
    pdl_enter();
    const uint32_t p0 = kPer * (blockIdx.x * blockDim.x + threadIdx.x);
    if (p0 >= b.npix)
        return;
    const uint32_t cnt = min(kPer, b.npix - p0);
    const bool whole = kPer == 4u && cnt == 4u;
    unsigned long long key[kPer], all = ~0ull;
    if (whole)
    {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(b.pix_key + p0);
        const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(b.pix_key + p0 + 2);
        const unsigned long long ks[4] = {a.x, a.y, c.x, c.y};
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u)
            key[u] = ks[u];
    }
    else
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u)
            key[u] = (u < cnt) ? b.pix_key[p0 + u] : ~0ull;
    int32_t map[4] = {-1, -1, -1, -1};
    uint8_t state[4] = {PX_EMPTY, PX_EMPTY, PX_EMPTY, PX_EMPTY};
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u)
        all &= key[u];
    if (all != ~0ull)
    {
        const int s0 = scan_of_pix(b, p0);
        const bool one = kPer == 1u || s0 + 1 >= b.nscan || p0 + kPer - 1u < b.scans[s0 + 1].pix_off; // all of scan s0
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u)
            if (key[u] != ~0ull)
            {
                const ScanDev& sd = b.scans[one ? s0 : scan_of_pix(b, p0 + u)];
                if (kPacked)
                {
                    map[u] = static_cast<int32_t>((static_cast<uint32_t>(key[u]) & ((1u << sd.key_cell) - 1u)) >> 1);
                    state[u] = (key[u] & 1ull) ? PX_OBSTACLE : PX_GROUND;
                }
                else
                {
                    map[u] = static_cast<int32_t>(static_cast<uint32_t>(key[u]));
                    state[u] = (b.pt_label[sd.pt_off + static_cast<uint32_t>(map[u])] == LP_LABEL_GROUND) ? PX_GROUND : PX_OBSTACLE;
                }
            }
    }
    if (whole)
    {
        *reinterpret_cast<int4*>(b.pix_map + p0) = make_int4(map[0], map[1], map[2], map[3]);
        *reinterpret_cast<uchar4*>(b.pix_state + p0) = make_uchar4(state[0], state[1], state[2], state[3]);
        return;
    }
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u)
        if (u < cnt)
        {
            b.pix_map[p0 + u] = map[u];
            b.pix_state[p0 + u] = state[u];
        }
}

// ------------------------------------------------------------------------------------------
// Dilation of the obstacle channel by a 5x5 rectangle clipped at the image border, and the
// row-major intersection queue (segmenter.cpp:486-514): one block per image row.
// ------------------------------------------------------------------------------------------
// Bit-mask form: a warp takes 32 consecutive pixels at a time; a ballot over each of the five
// rows h-2..h+2 gives the obstacle bits of that segment, the rows are OR-ed, and the +-2 column
// dilation is done with shifts, the two halo bits on each side coming from the neighbouring
// segments (zero outside the image: the rectangle is clipped at the border). Dilation changes
// only ground and empty pixels, never the obstacle channel, so rows are independent. Each warp
// walks a contiguous run of segments; the queue keeps column order through per-warp counts.
constexpr int kRowWords = 2048; // 32-column words of the widest image row (65,535 columns)
__global__ void __launch_bounds__(256) k_dilate_rows(BatchDev b)
{
    pdl_enter();
    __shared__ uint32_t wcount[8];
    __shared__ uint32_t woff[8];
    __shared__ uint32_t bits[kRowWords + 2], queued[kRowWords];
    const uint32_t r = blockIdx.x;
    const int s = scan_of_row(b, r);
    const ScanDev& sd = b.scans[s];
    const int32_t h = static_cast<int32_t>(r - sd.row_off);
    const int32_t H = sd.H, W = sd.W;
    uint8_t* st = b.pix_state + sd.pix_off;
    const uint32_t row_base = sd.pix_off + static_cast<uint32_t>(h * W);
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const int32_t nseg = (W + 31) / 32;
    const int32_t per = (nseg + 7) / 8;
    const int32_t s0 = static_cast<int32_t>(warp) * per, s1 = min(nseg, s0 + per);
    // the obstacles of the rows h - 2 .. h + 2, a bit per column, four words' loads in flight
    for (int32_t g = s0; g < s1; g += 4)
    {
        bool any[4];
#pragma unroll
        for (int32_t u = 0; u < 4; ++u)
        {
            const int32_t w = (g + u) * 32 + static_cast<int32_t>(lane);
            any[u] = false;
#pragma unroll
            for (int32_t dh = -2; dh <= 2; ++dh)
                any[u] |= g + u < s1 && w < W && h + dh >= 0 && h + dh < H && st[(h + dh) * W + w] == PX_OBSTACLE;
        }
#pragma unroll
        for (int32_t u = 0; u < 4; ++u)
        {
            const uint32_t m = __ballot_sync(0xffffffffu, any[u]);
            if (lane == 0 && g + u < s1)
                bits[g + u + 1] = m;
        }
    }
    if (threadIdx.x == 0)
        bits[0] = bits[nseg + 1] = 0u;
    __syncthreads();
    // pass 1: dilate, update the states, count the queued (ground -> intersection) pixels
    uint32_t count = 0u;
    for (int32_t g = s0; g < s1; g += 4)
    {
        uint8_t c[4];
#pragma unroll
        for (int32_t u = 0; u < 4; ++u)
        {
            const int32_t seg = min(g + u, nseg - 1), w = seg * 32 + static_cast<int32_t>(lane);
            const uint32_t left = bits[seg], cur = bits[seg + 1], right = bits[seg + 2];
            const uint32_t d = cur | (cur << 1) | (cur << 2) | (cur >> 1) | (cur >> 2) | (left >> 31) | (left >> 30) |
                               (right << 31) | (right << 30);
            c[u] = (g + u < s1 && w < W && ((d >> lane) & 1u)) ? st[h * W + w] : static_cast<uint8_t>(PX_OBSTACLE);
        }
#pragma unroll
        for (int32_t u = 0; u < 4; ++u)
        {
            const int32_t w = (g + u) * 32 + static_cast<int32_t>(lane);
            if (c[u] == PX_GROUND)
                st[h * W + w] = PX_INTERSECT;
            else if (c[u] == PX_EMPTY)
                st[h * W + w] = PX_EMPTY_RED;
            const uint32_t m = __ballot_sync(0xffffffffu, c[u] == PX_GROUND);
            if (lane == 0 && g + u < s1)
                queued[g + u] = m;
            count += static_cast<uint32_t>(__popc(m));
        }
    }
    if (lane == 0)
        wcount[warp] = count;
    __syncthreads();
    __shared__ uint32_t qbase;
    if (threadIdx.x == 0)
    {
        uint32_t run = 0u;
        for (int k = 0; k < 8; ++k)
        {
            woff[k] = run;
            run += wcount[k];
        }
        b.row_cnt[r] = run;
        // the row's segment of the scan's queue; the capacity bound (a queued pixel holds a point)
        // cannot be exceeded, checked all the same
        qbase = run ? atomicAdd(&b.state[s].n_queue, run) : 0u;
        if (qbase + run > sd.jq_cap)
        {
            raise_err(&b.state[s], ERR_INTERNAL);
            b.row_cnt[r] = 0u;
            atomicSub(&b.state[s].n_queue, run);
            qbase = 0xffffffffu;
        }
    }
    __syncthreads();
    // pass 2: queue entries in column order
    uint32_t pos = woff[warp];
#pragma unroll 4
    for (int32_t seg = s0; seg < s1; ++seg)
    {
        const int32_t w = seg * 32 + static_cast<int32_t>(lane);
        const uint32_t m = queued[seg];
        const bool inter = ((m >> lane) & 1u) != 0u;
        if (inter)
        {
            const uint32_t j = pos + static_cast<uint32_t>(__popc(m & ((1u << lane) - 1u)));
            b.row_cols[row_base + j] = static_cast<uint16_t>(w);
            // (row, position | column << 16, the pixel's point): the weights pass starts here; the
            // depth key, no longer needed, takes the pixel's queue index for those that read its outcome
            if (qbase != 0xffffffffu)
            {
                b.jq[sd.jq_off + qbase + j] = make_uint4(r, j | (static_cast<uint32_t>(w) << 16),
                                                         static_cast<uint32_t>(b.pix_map[row_base + static_cast<uint32_t>(w)]), 0u);
                b.pix_depth[row_base + static_cast<uint32_t>(w)] = qbase + j;
            }
        }
        pos += static_cast<uint32_t>(__popc(m));
    }
}

// Offsets of the 24-neighbour kernel (segmenter.cpp:527-530: the 5x5 window without its centre,
// row-major) as arithmetic on the slot index (folds to constants in unrolled loops).
__device__ __forceinline__ constexpr int32_t jcp_dh(int k)
{
    return k < 10 ? -2 + k / 5 : (k < 14 ? 0 : 1 + (k - 14) / 5);
}
__device__ __forceinline__ constexpr int32_t jcp_dw(int k)
{
    return k < 10 ? k % 5 - 2 : (k < 14 ? (k < 12 ? k - 12 : k - 11) : (k - 14) % 5 - 2);
}

__device__ __forceinline__ uint8_t final_view(uint8_t st)
{
    return (st == PX_GROUND || st == PX_RES_G) ? V_G : ((st == PX_OBSTACLE || st == PX_RES_O) ? V_O : V_U);
}
__device__ __forceinline__ uint8_t pre_view(uint8_t st)
{
    return (st == PX_GROUND) ? V_G : ((st == PX_OBSTACLE) ? V_O : V_U);
}

// ------------------------------------------------------------------------------------------
// The vote of the queued pixels (segmenter.cpp:523-637). The reference takes them in row-major
// order, in place: a pixel reads the final colours of queued pixels above it and to its left in its
// row (kernel slots 0-11), pre-vote colours everywhere else. The sums run in slot order: a neighbour
// labelled ground adds its normalised weight to g, one labelled obstacle to o, and the pixel becomes
// an obstacle iff o > g.
//
// Taking image rows one after the other (one CTA per scan, the row as a scan of transition maps)
// made the vote the longest kernel of every call: a chain of 64-128 rows at 2 us each. But most
// outcomes do not depend on their open neighbours: weights are never negative and rounding is
// monotone, so with every open neighbour counted to o and none to g (and the other way round) the
// same chain of additions bounds o and g for any outcome of theirs. A pixel whose bounds do not
// overlap is decided at once, in any order, with the reference's result. k_jcp_weights decides about
// half of the pixels this way, in parallel; k_jcp_resolve repeats the test for the rest as their
// neighbours are decided (about 20-100 hops instead of one step per row; every hop decides at
// least the first open pixel in the reference's order).
// ------------------------------------------------------------------------------------------
enum : uint32_t
{
    JST_OPEN = 3u // queued pixel not decided yet (V_U, V_G, V_O otherwise)
};

// Decision from the normalised weights and the slots' labels (bit 0 of slot k's label in m0, bit 1 in
// m1; both: the slot is open). V_G / V_O, or JST_OPEN while the open slots could change it.
__device__ __forceinline__ uint32_t vote_bounds(const float* wn, uint32_t m0, uint32_t m1)
{
    float2 lo = make_float2(0.0F, 0.0F), hi = lo; // (g, o) without the open slots, with them on both sides
    const uint32_t g = m0 & ~m1, o = m1 & ~m0;
#pragma unroll
    for (int k = 0; k < 24; ++k)
    {
        const uint32_t bit = 1u << k;
        lo = __fadd2_rn(lo, make_float2((g & bit) ? wn[k] : 0.0F, (o & bit) ? wn[k] : 0.0F));
        hi = __fadd2_rn(hi, make_float2((m0 & bit) ? wn[k] : 0.0F, (m1 & bit) ? wn[k] : 0.0F));
    }
    if ((m0 & m1) == 0u)
        return (lo.y > lo.x) ? V_O : V_G;
    if (lo.y > hi.x)
        return V_O; // o >= lo.y > hi.x >= g
    return (hi.y <= lo.x) ? V_G : JST_OPEN; // o <= hi.y <= lo.x <= g (false for nan weights: they stay open)
}

// Records of the open pixels, by list position (fields of 16 bytes, jq_total entries each):
// 0-5 the 24 normalised weights; 6-8 for slots 0-11 the queue index behind an open slot, else
// kDepFixed | label; 9 (label bit 0 per slot, label bit 1 per slot, queue index, weight sum).
constexpr uint32_t kDepFixed = 0x80000000u;

__device__ __forceinline__ uint4& jrec(const BatchDev& b, uint32_t field, uint32_t at)
{
    return b.jrec[static_cast<size_t>(field) * b.jq_total + at];
}

// Weights of the queued pixels (segmenter.cpp:545-607): 0 for an empty neighbour or one farther than
// the kernel threshold, else expf(-amp * dist). A warp takes up to 32 consecutive pixels of a scan's
// queue: lane k = kernel slot k for the gathers (four pixels side by side), the weights and the
// divisions by the sum, lane = pixel for the sums (slot order, as the reference's loop adds them) and
// the decision. Fewer pixels per warp where the queues would leave warps idle (4 to 32, from their
// total). The exponential and the division stand in loops that are not unrolled: on a single scan
// every warp runs this code once, and fetching it is most of the time.
// Only open pixels leave a record. A pixel whose window leaves the image is completed by
// k_jcp_resolve: such a slot keeps what an earlier queued pixel left there; the raw weights of each
// row's last three queued pixels, the only ones read for that, go to jw.
struct JcpTile // a warp's pixels
{
    float w[32][25]; // squared distances, then weights, then normalised weights
    float sum[32];
    uint32_t dep[32][13];
    uint32_t m0[32], m1[32], oob[32], valid[32];
};
constexpr uint32_t kWeightThreads = 128;

__global__ void __launch_bounds__(kWeightThreads) k_jcp_weights(BatchDev b)
{
    pdl_enter();
    __shared__ JcpTile tiles[kWeightThreads / 32];
    const uint32_t lane = lane_id();
    const int k = static_cast<int>(lane);
    const int32_t dh = jcp_dh(k), dw = jcp_dw(k);
    JcpTile& t = tiles[threadIdx.x >> 5];
    const uint32_t nwarp = gridDim.x * (kWeightThreads / 32u);
    uint32_t total = 0u;
    for (int q = 0; q < b.nscan; ++q)
        total += b.state[q].n_queue;
    const uint32_t per = min(32u, 4u * max(1u, div_up(total, 4u * nwarp))); // pixels per warp and turn
    int s = 0; // the cursor: scan s owns turns [tbase, tbase + div_up(nq, per))
    uint32_t tbase = 0u, nq = b.nscan > 0 ? b.state[0].n_queue : 0u;
    for (uint32_t it = (blockIdx.x * kWeightThreads + threadIdx.x) >> 5;; it += nwarp)
    {
        while (s < b.nscan && it >= tbase + div_up(nq, per))
        {
            tbase += div_up(nq, per);
            ++s;
            nq = (s < b.nscan) ? b.state[s].n_queue : 0u;
        }
        if (s >= b.nscan)
            break; // uniform over the warp
        const ScanDev& sd = b.scans[s];
        const uint32_t q0 = (it - tbase) * per;
        const uint32_t cnt = min(per, nq - q0);
        const int32_t H = sd.H, W = sd.W;
        const int32_t* map = b.pix_map + sd.pix_off;
        const uint32_t* qidx = b.pix_depth + sd.pix_off;
        const uint8_t* st = b.pix_state + sd.pix_off;
        const float4* pts = b.pts + sd.pt_off;
        const float kthr2 = sd.kthr2, namp = -sd.amp;
        const uint4 mine_e = b.jq[sd.jq_off + q0 + min(lane, cnt - 1u)]; // lane p: pixel p's queue entry
        const uint32_t mine_m = b.row_cnt[mine_e.x];
        for (uint32_t p0 = 0; p0 < cnt; p0 += 4u)
        {
            int32_t ni[4];
            uint8_t ns[4];
            uint32_t qi[4];
            float4 cp[4], np[4];
            bool inb[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
            {
                const int src = static_cast<int>(min(p0 + u, cnt - 1u));
                const int32_t h = static_cast<int32_t>(__shfl_sync(0xffffffffu, mine_e.x, src) - sd.row_off);
                const int32_t w = static_cast<int32_t>(__shfl_sync(0xffffffffu, mine_e.y, src) >> 16);
                const int32_t hh = h + dh, ww = w + dw;
                inb[u] = k < 24 && hh >= 0 && hh < H && ww >= 0 && ww < W;
                const int32_t at = inb[u] ? hh * W + ww : 0;
                ni[u] = inb[u] ? map[at] : -1;
                ns[u] = st[at];
                qi[u] = (k < 12) ? qidx[at] : 0u;
                cp[u] = pts[__shfl_sync(0xffffffffu, mine_e.z, src)];
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
                np[u] = (ni[u] >= 0) ? pts[ni[u]] : cp[u];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
            {
                const uint32_t p = p0 + u;
                const float dx = cp[u].x - np[u].x;
                const float dy = cp[u].y - np[u].y;
                const float dz = cp[u].z - np[u].z;
                const float d2 = dx * dx + dy * dy + dz * dz;
                // slots 12-23 are not voted before this pixel
                const uint32_t code = (k < 12 && ns[u] == PX_INTERSECT) ? 3u : pre_view(ns[u]);
                const uint32_t va = __ballot_sync(0xffffffffu, ni[u] >= 0 && !(d2 > kthr2));
                const uint32_t c0 = __ballot_sync(0xffffffffu, code & 1u), c1 = __ballot_sync(0xffffffffu, code & 2u);
                const uint32_t ob = __ballot_sync(0xffffffffu, k < 24 && !inb[u]);
                if (p < cnt)
                {
                    if (k < 24)
                        t.w[p][k] = d2;
                    if (k < 12) // the queue index behind an open slot, else its label
                        t.dep[p][k] = (code == 3u) ? qi[u] : kDepFixed | code;
                    if (lane == 0)
                    {
                        t.m0[p] = c0;
                        t.m1[p] = c1;
                        t.oob[p] = ob;
                        t.valid[p] = va;
                    }
                }
            }
        }
        __syncwarp();
#pragma unroll 1
        for (uint32_t p = 0; p < cnt; ++p)
        {
            float wt = 0.0F;
            if ((t.valid[p] >> k) & 1u)
                wt = lpm::cr_expf(namp * sqrtf(t.w[p][k]));
            const uint32_t nz = __ballot_sync(0xffffffffu, wt != 0.0F);
            if (k < 24)
                t.w[p][k] = wt;
            if (k < 12 && wt == 0.0F)
                t.dep[p][k] = kDepFixed | V_U;
            if (lane == 0) // a slot without weight has no label
            {
                t.m0[p] &= nz;
                t.m1[p] &= nz;
            }
        }
        __syncwarp();
        const uint32_t p = min(lane, cnt - 1u);
        const bool mine = lane < cnt;
        float wn[24];
        float sum = 0.0F;
#pragma unroll
        for (int q = 0; q < 24; ++q)
        {
            wn[q] = t.w[p][q];
            sum += wn[q];
        }
        const uint32_t j = mine_e.y & 0xffffu;
        if (mine && j + 3u >= mine_m)
        {
            float4* raw = reinterpret_cast<float4*>(b.jw + (static_cast<size_t>(mine_e.x) * 3u + (j + 3u - mine_m)) * kJwStride);
#pragma unroll
            for (int q = 0; q < 6; ++q)
                raw[q] = make_float4(wn[4 * q], wn[4 * q + 1], wn[4 * q + 2], wn[4 * q + 3]);
        }
        if (mine)
            t.sum[lane] = sum;
        __syncwarp();
#pragma unroll 1
        for (uint32_t p1 = 0; p1 < cnt; ++p1)
        {
            const float sp = t.sum[p1];
            if (k < 24)
                t.w[p1][k] = (fabsf(sp) > FLT_EPSILON) ? t.w[p1][k] / sp : 0.0F;
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 24; ++q)
            wn[q] = t.w[p][q];
        const uint32_t m0 = t.m0[p], m1 = t.m1[p];
        const bool border = t.oob[p] != 0u;
        uint32_t x = JST_OPEN;
        if (!(fabsf(sum) > FLT_EPSILON))
            x = V_U; // keeps the queue's colour
        else if (!border)
            x = vote_bounds(wn, m0, m1);
        if (mine)
            b.jst[sd.jq_off + q0 + lane] = static_cast<uint8_t>(x);
        const bool open = mine && x == JST_OPEN;
        const uint32_t om = __ballot_sync(0xffffffffu, open);
        uint32_t slot = 0u;
        if (om && lane == 0)
            slot = atomicAdd(&b.state[s].n_open, static_cast<uint32_t>(__popc(om)));
        slot = __shfl_sync(0xffffffffu, slot, 0) + static_cast<uint32_t>(__popc(om & ((1u << lane) - 1u)));
        if (open)
        {
            const uint32_t r = sd.jq_off + slot;
#pragma unroll
            for (uint32_t f = 0; f < 6; ++f)
                jrec(b, f, r) = make_uint4(__float_as_uint(wn[4 * f]), __float_as_uint(wn[4 * f + 1]),
                                           __float_as_uint(wn[4 * f + 2]), __float_as_uint(wn[4 * f + 3]));
#pragma unroll
            for (uint32_t f = 0; f < 3; ++f)
                jrec(b, 6u + f, r) = make_uint4(t.dep[p][4 * f], t.dep[p][4 * f + 1], t.dep[p][4 * f + 2], t.dep[p][4 * f + 3]);
            jrec(b, 9u, r) = make_uint4(m0, m1, q0 + lane, __float_as_uint(sum));
            if (border)
                b.jborder[sd.jq_off + atomicAdd(&b.state[s].n_border, 1u)] = slot;
        }
        __syncwarp(); // the tile is read before the next turn fills it
    }
}

// What the reference's weight and label buffer holds for slot k (dh, dw) of a pixel of row h whose
// slot lies outside the image (segmenter.cpp:552-556): the values of the last earlier queued pixel
// with that slot inside. Right of the image that can be a pixel of the same row (columns up to
// W - 1 - dw); otherwise it lies in the nearest earlier row that has one. Among a row's queued pixels
// it is one of the last three (at most two columns lie beyond W - 1 - dw).
__device__ __forceinline__ bool stale_slot(const BatchDev& b, const ScanDev& sd, int k, int32_t h, float& w, uint32_t& code,
                                           uint32_t& dep)
{
    const int32_t dh = jcp_dh(k), dw = jcp_dw(k);
    const int32_t H = sd.H, W = sd.W;
    const uint8_t* st = b.pix_state + sd.pix_off;
    w = 0.0F;
    code = V_U;
    dep = 0u;
    for (int32_t r = (dw > 0 && h + dh >= 0 && h + dh < H) ? h : h - 1; r >= 0; --r)
    {
        const int32_t m = static_cast<int32_t>(b.row_cnt[sd.row_off + static_cast<uint32_t>(r)]);
        const int32_t hh = r + dh;
        if (m == 0 || hh < 0 || hh >= H)
            continue;
        const uint16_t* cols = b.row_cols + sd.pix_off + static_cast<uint32_t>(r * W);
        const int32_t lim = W - 1 - (dw > 0 ? dw : 0);
        int32_t j = m - 1;
        while (j >= 0 && j >= m - 3 && static_cast<int32_t>(cols[j]) > lim)
            --j;
        if (j < 0 || j < m - 3 || static_cast<int32_t>(cols[j]) + dw < 0)
            continue; // no queued pixel of this row has the slot inside
        w = b.jw[(static_cast<size_t>(sd.row_off + static_cast<uint32_t>(r)) * 3u + static_cast<uint32_t>(j + 3 - m)) * kJwStride + k];
        if (w != 0.0F)
        {
            const uint32_t addr = static_cast<uint32_t>(hh * W + static_cast<int32_t>(cols[j]) + dw);
            if (k < 12 && st[addr] == PX_INTERSECT)
            {
                code = 3u; // that pixel's outcome
                dep = b.pix_depth[sd.pix_off + addr];
            }
            else
                code = pre_view(st[addr]);
        }
        return true;
    }
    return false;
}

// The open pixels of a scan, one cluster of kCtas CTAs each: the border pixels' stale slots
// first, then (more open pixels than threads only) rounds over the list, then every thread watches
// its own pixel's open neighbours and repeats the test when one is decided. Each CTA keeps every
// queued pixel's state in its shared memory and a decision is written into all of them, so
// watching costs local reads only (scans of more than `cap` queued pixels watch global memory). What
// neither decides within its budget is left to vote_rows.
// Bound by the chain of hops, about 700 cycles each. Chains of pixels of one row, each hanging on the
// one to its left, would make 60 hops on a 64 x 2048 scan and 130 on a 32 x 4096 one: where the
// bounds show that one open neighbour alone decides (it on ground: ground, it on obstacle: obstacle,
// whatever the others become), the pixel becomes a copy of that neighbour, and copies of copies
// skip ahead, so the hops of a chain grow with its logarithm (15 and 29 hops).
// Several CTAs because a hop's price grows with the warps that share an SM, and because the rounds
// read 160 bytes per open pixel. 8 for launches of up to kResolveWide scans (28 us on a 64 x 2048
// scan, 68 us on six mixed ones; 4 CTAs: 31 and 107 us; one CTA without copies: 102 and 417 us; the
// row-by-row kernel: 126 and 182 us), 4 for more, whose clusters take the SMs from the other parts of a
// split batch (64-scan batch, eight parts: 1.92 ms against 1.97 ms with 8).
constexpr uint32_t kResolveThreads = 512;
constexpr uint32_t kResolveStates = 24u * 1024u; // queued pixels whose states fit shared memory (4 bytes each)
constexpr int kResolveWide = 7;           // scans of a launch up to which a scan takes 8 CTAs
// A round takes as long as it has open pixels, and where they hang on one another in chains as long as the image it
// decides little more than one pixel of each. So rounds (2 us for 4,096 pixels) and watching end where they
// have cost about what vote_rows would (2 us for every row and 512 pixels). Stripes over a 64 x 2048 and a 128 x 4096
// image: 1.1 and 4.3 ms, against 1,276 and 16,000 without an end. The workloads' scans stay below it; with half of
// this budget one scan each of two 64-scan batches did not (107 -> 146 us; 1.79 -> 1.80 ms a batch).
constexpr uint32_t kSpinsLocal = 32, kSpinsGlobal = 4; // polls of a pixel's neighbours for each step of vote_rows

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of this CTA's shared variable p in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_smem(const void* p, uint32_t rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
    return a;
}

__device__ __forceinline__ uint32_t jrec_load(const BatchDev& b, uint32_t r, float* wn, uint32_t* dep, uint32_t& m0, uint32_t& m1)
{
#pragma unroll
    for (uint32_t f = 0; f < 6; ++f)
    {
        const uint4 v = jrec(b, f, r);
        wn[4 * f] = __uint_as_float(v.x);
        wn[4 * f + 1] = __uint_as_float(v.y);
        wn[4 * f + 2] = __uint_as_float(v.z);
        wn[4 * f + 3] = __uint_as_float(v.w);
    }
#pragma unroll
    for (uint32_t f = 0; f < 3; ++f)
    {
        const uint4 v = jrec(b, 6u + f, r);
        dep[4 * f] = v.x;
        dep[4 * f + 1] = v.y;
        dep[4 * f + 2] = v.z;
        dep[4 * f + 3] = v.w;
    }
    const uint4 v = jrec(b, 9u, r);
    m0 = v.x;
    m1 = v.y;
    return v.z;
}

// An entry in shared memory: the state in the lower half (label bit 0 at bit 0, label bit 1 at bit
// 12, so that twelve of them shift and add into the two label masks of slots 0-11), in the upper half
// the queue index + 1 of the pixel it copies. The last three entries are the labels themselves, for
// the slots that are not open.
__device__ __forceinline__ uint32_t wide_state(uint32_t v)
{
    return (v & 1u) | ((v >> 1) << 12);
}

// What rounds and watching leave open, by one CTA, row by row as the reference goes: with the rows above decided, a
// pixel's outcome depends on its two neighbours to the left alone (kernel slots 10 and 11, at most two
// places back in the queue), so it is a map of the last two outcomes onto the next two, and the maps
// of 512 pixels are composed by a scan.
struct RowVote // of one scan
{
    volatile uint8_t* st;  // outcomes by queue index
    const uint32_t* slot;  // record of each open pixel
    const uint4* rec;      // field f of record r at rec[f * stride + r]
    size_t stride;
    const uint32_t* cnt;   // queued pixels of each row
    const uint16_t* cols;  // their columns
    const uint32_t* qidx;  // queue index by pixel
    int32_t H, W;
};

// A map of the state (outcome before last, last outcome; 1: obstacle): two bits of the next state for each.
__device__ __forceinline__ uint32_t then_map(uint32_t first, uint32_t second)
{
    uint32_t r = 0u;
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u)
        r |= ((second >> (2u * ((first >> (2u * u)) & 3u))) & 3u) << (2u * u);
    return r;
}

__device__ __noinline__ void vote_rows(const RowVote v)
{
    constexpr uint32_t kSame = 0xe4u; // the identity
    __shared__ uint32_t total[kResolveThreads / 32];
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    for (int32_t h = 0; h < v.H; ++h)
    {
        const uint32_t m = v.cnt[h];
        const uint32_t q0 = m ? v.qidx[h * v.W + v.cols[h * v.W]] : 0u; // the row's queue entries lie behind one another
        for (uint32_t j0 = 0; j0 < m; j0 += kResolveThreads)
        {
            const uint32_t q = q0 + j0 + tid;
            const uint32_t is = (j0 + tid < m) ? v.st[q] : V_U;
            const bool open = is == JST_OPEN;
            if (!__syncthreads_or(open))
                continue;
            uint32_t map = (j0 + tid < m) ? (is == V_O ? 0xddu : 0x88u) : kSame; // decided: (., x) -> (x, outcome)
            if (open)
            {
                const uint4* rec = v.rec + __ldcg(&v.slot[q]);
                float wn[24];
#pragma unroll
                for (uint32_t f = 0; f < 6; ++f)
                {
                    const uint4 w = rec[f * v.stride];
                    wn[4 * f] = __uint_as_float(w.x);
                    wn[4 * f + 1] = __uint_as_float(w.y);
                    wn[4 * f + 2] = __uint_as_float(w.z);
                    wn[4 * f + 3] = __uint_as_float(w.w);
                }
                const uint4 masks = rec[9u * v.stride];
                uint32_t m0 = masks.x & 0xfff000u, m1 = masks.y & 0xfff000u;
                uint32_t last = 0u, before = 0u; // slots that read the last outcome, the one before
#pragma unroll
                for (uint32_t f = 0; f < 3; ++f)
                {
                    const uint4 d4 = rec[(6u + f) * v.stride];
                    const uint32_t d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u)
                    {
                        const uint32_t k = 4u * f + u;
                        const uint32_t x = (d[u] & kDepFixed) ? d[u] & 3u : v.st[d[u]];
                        if (x != JST_OPEN)
                        {
                            m0 |= (x & 1u) << k;
                            m1 |= (x >> 1) << k;
                        }
                        else if (q - d[u] == 1u)
                            last |= 1u << k;
                        else
                            before |= 1u << k;
                    }
                }
                // the sums of slots 0-9 once, the others for every state (vote_bounds for a known state, its terms in the same order)
                auto term = [&](uint32_t k, uint32_t g, uint32_t o) {
                    return make_float2(((g >> k) & 1u) ? wn[k] : 0.0F, ((o >> k) & 1u) ? wn[k] : 0.0F);
                };
                float2 head = make_float2(0.0F, 0.0F); // (ground, obstacle)
#pragma unroll
                for (uint32_t k = 0; k < 10; ++k)
                    head = __fadd2_rn(head, term(k, m0, m1));
                map = 0u;
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u)
                {
                    const uint32_t o = ((u & 1u) ? last : 0u) | ((u & 2u) ? before : 0u); // these on obstacle
                    float2 sum = head;
#pragma unroll
                    for (uint32_t k = 10; k < 24; ++k)
                        sum = __fadd2_rn(sum, term(k, m0 | ((last | before) & ~o), m1 | o));
                    map |= (((u & 1u) << 1) | (sum.y > sum.x ? 1u : 0u)) << (2u * u);
                }
            }
            uint32_t incl = map;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t below = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= static_cast<uint32_t>(o))
                    incl = then_map(below, incl);
            }
            if (lane == 31u)
                total[warp] = incl;
            __syncthreads();
            uint32_t state = 0u; // (an open pixel never reads outcomes of the step before: those are decided)
            for (uint32_t w = 0; w < warp; ++w)
                state = (total[w] >> (2u * state)) & 3u;
            state = (incl >> (2u * state)) & 3u;
            if (open)
                v.st[q] = static_cast<uint8_t>((state & 1u) ? V_O : V_G);
            __syncthreads();
        }
    }
}

template <uint32_t kCtas>
__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(kResolveThreads) k_jcp_resolve(BatchDev b, uint32_t cap)
{
    pdl_enter();
    constexpr uint32_t kAll = kResolveThreads * kCtas;
    extern __shared__ __align__(16) uint32_t sst[]; // cap + 4 entries
    __shared__ uint32_t s_n[2]; // pixels left open by a round (of the cluster's first CTA), alternating
    __shared__ uint32_t s_left; // pixels remain for vote_rows (of the cluster's first CTA)
    const int s = static_cast<int>(blockIdx.x / kCtas);
    const uint32_t rank = blockIdx.x % kCtas;
    const ScanDev& sd = b.scans[s];
    const uint32_t nq = b.state[s].n_queue, nopen = b.state[s].n_open, nborder = b.state[s].n_border;
    if (nopen == 0u)
        return;
    const uint32_t tid = threadIdx.x, lane = lane_id();
    const uint32_t warp = (tid >> 5) * kCtas + rank; // warp and thread of the cluster: neighbouring
    const uint32_t all = warp * 32u + lane;                 // warps on different SMs
    uint8_t* gst = b.jst + sd.jq_off;
    const bool local = nq <= cap;
    if (local)
    {
        for (uint32_t i = tid; i < (nq + 3u) / 4u; i += kResolveThreads) // jq_off is a multiple of 16, the array padded
        {
            const uint32_t v = reinterpret_cast<const uint32_t*>(gst)[i];
            reinterpret_cast<uint4*>(sst)[i] = make_uint4(wide_state(v & 3u), wide_state((v >> 8) & 3u),
                                                          wide_state((v >> 16) & 3u), wide_state((v >> 24) & 3u));
        }
        if (tid < 3u)
            sst[cap + tid] = wide_state(tid);
    }
    for (uint32_t i = warp; i < nborder; i += kAll / 32u)
    {
        const uint32_t r = sd.jq_off + b.jborder[sd.jq_off + i];
        const uint4 rec = jrec(b, 9u, r);
        const uint4 e = b.jq[sd.jq_off + rec.z];
        const int k = static_cast<int>(lane);
        const int32_t h = static_cast<int32_t>(e.x - sd.row_off), hh = h + jcp_dh(k);
        const int32_t ww = static_cast<int32_t>(e.y >> 16) + jcp_dw(k);
        const bool oob = k < 24 && !(hh >= 0 && hh < sd.H && ww >= 0 && ww < sd.W);
        uint32_t code = ((rec.x >> k) & 1u) | (((rec.y >> k) & 1u) << 1);
        if (oob)
        {
            float w;
            uint32_t dep;
            stale_slot(b, sd, k, h, w, code, dep);
            reinterpret_cast<float*>(&jrec(b, static_cast<uint32_t>(k) / 4u, r))[k & 3] = w / __uint_as_float(rec.w);
            if (k < 12)
                reinterpret_cast<uint32_t*>(&jrec(b, 6u + static_cast<uint32_t>(k) / 4u, r))[k & 3] =
                    (code == 3u) ? dep : kDepFixed | code;
        }
        const uint32_t m0 = __ballot_sync(0xffffffffu, code & 1u), m1 = __ballot_sync(0xffffffffu, code & 2u);
        if (lane == 0)
            jrec(b, 9u, r) = make_uint4(m0, m1, rec.z, rec.w);
    }
    if (tid < 2u)
        s_n[tid] = 0u;
    if (tid == 2u)
        s_left = 0u;
    __threadfence();
    cluster_barrier();
    const uint32_t n_addr[2] = {peer_smem(&s_n[0], 0u), peer_smem(&s_n[1], 0u)};
    uint32_t peer[kCtas];
#pragma unroll
    for (uint32_t c = 0; c < kCtas; ++c)
        peer[c] = peer_smem(sst, c);
    const uint32_t own = smem_addr(sst);
    auto tell = [&](uint32_t at, uint32_t v) { // 16 bits at byte offset `at` of every CTA's entries
#pragma unroll
        for (uint32_t c = 0; c < kCtas; ++c)
            asm volatile("st.volatile.shared::cluster.u16 [%0], %1;" ::"r"(peer[c] + at), "h"(static_cast<uint16_t>(v)) : "memory");
    };
    auto watch = [&](uint32_t addr) -> uint32_t {
        uint16_t v;
        asm volatile("ld.volatile.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
        return v;
    };
    auto decide = [&](uint32_t q, uint32_t x) {
        if (local)
            tell(4u * q, wide_state(x));
        else
            *(reinterpret_cast<volatile uint8_t*>(gst) + q) = static_cast<uint8_t>(x);
    };
    // dep[0..11] (record fields 6-8) as what `labels` reads: shared-memory addresses, or indices
    auto locate = [&](uint32_t* dep) {
#pragma unroll
        for (int k = 0; k < 12; ++k)
            if (local)
                dep[k] = own + 4u * ((dep[k] & kDepFixed) ? cap + (dep[k] & 3u) : dep[k]);
    };
    // the labels of slots 0-11 now: bit 0 of each in bits 0-11, bit 1 in bits 12-23
    auto labels = [&](const uint32_t* dep) {
        uint32_t acc = 0u;
        if (local)
        {
#pragma unroll
            for (int k = 0; k < 12; ++k)
                acc += watch(dep[k]) << k;
        }
        else
        {
#pragma unroll
            for (int k = 0; k < 12; ++k)
                acc += wide_state((dep[k] & kDepFixed) ? dep[k] & 3u
                                                       : *(reinterpret_cast<volatile uint8_t*>(gst) + dep[k])) << k;
        }
        return acc;
    };
    auto vote = [&](const float* wn, uint32_t acc, uint32_t m0, uint32_t m1) {
        return vote_bounds(wn, (m0 & 0xfff000u) | (acc & 0xfffu), (m1 & 0xfff000u) | (acc >> 12));
    };
    float wn[24];
    uint32_t dep[12], m0, m1;
    uint32_t n = nopen;
    uint32_t *cur = nullptr, *next = b.jlist + sd.jq_off, *other = b.jlist + b.jq_total + sd.jq_off; // null: all positions
    const uint32_t steps = static_cast<uint32_t>(sd.H) + nq / kResolveThreads; // of vote_rows
    uint32_t spent = 0u;
    for (uint32_t round = 0; n > kAll && spent <= steps; ++round)
    {
        spent += 1u + n / (8u * kResolveThreads);
        const uint32_t cnt = n_addr[round & 1u];
        for (uint32_t t0 = warp * 32u; t0 < n; t0 += kAll)
        {
            const uint32_t t = t0 + lane;
            bool open = false;
            uint32_t at = 0u;
            if (t < n)
            {
                at = cur ? __ldcg(&cur[t]) : t;
                const uint32_t q = jrec_load(b, sd.jq_off + at, wn, dep, m0, m1);
                locate(dep);
                const uint32_t x = vote(wn, labels(dep), m0, m1);
                open = x == JST_OPEN;
                if (!open)
                {
                    decide(q, x);
                    gst[q] = static_cast<uint8_t>(x);
                }
            }
            const uint32_t mask = __ballot_sync(0xffffffffu, open);
            uint32_t base = 0u;
            if (lane == 0 && mask)
                asm volatile("atom.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(base) : "r"(cnt), "r"(__popc(mask)) : "memory");
            base = __shfl_sync(0xffffffffu, base, 0);
            if (open)
                next[base + static_cast<uint32_t>(__popc(mask & ((1u << lane) - 1u)))] = at;
        }
        __threadfence();
        cluster_barrier();
        uint32_t left;
        asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(left) : "r"(cnt) : "memory");
        if (all == 0u)
            s_n[(round & 1u) ^ 1u] = 0u; // the next round's count (its last readers passed the barrier above)
        cluster_barrier();
        n = left;
        cur = next;
        next = other;
        other = cur;
    }
    // what is left to vote_rows: its records by queue index
    auto leave = [&](uint32_t at, uint32_t q) {
        next[q] = at;
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_smem(&s_left, 0u)), "r"(1u) : "memory");
    };
    if (n > kAll)
    {
        for (uint32_t t = all; t < n; t += kAll)
        {
            const uint32_t at = cur ? __ldcg(&cur[t]) : t;
            leave(at, jrec(b, 9u, sd.jq_off + at).z);
        }
    }
    else if (all < n)
    {
        const uint32_t at = cur ? __ldcg(&cur[all]) : all;
        const uint32_t q = jrec_load(b, sd.jq_off + at, wn, dep, m0, m1);
        locate(dep);
        uint32_t x = JST_OPEN, seen = 0xffffffffu, copied = 0u; // copied: the entry this pixel copies
        const uint32_t spins = (local ? kSpinsLocal : kSpinsGlobal) * steps;
        for (uint32_t spin = 0; x == JST_OPEN && spin < spins; ++spin)
        {
            if (copied != 0u)
            {
                const uint32_t v = watch(copied), further = watch(copied + 2u);
                if (v != wide_state(JST_OPEN))
                    x = (v & 1u) ? V_G : V_O;
                else if (further != 0u)
                {
                    copied = own + 4u * (further - 1u);
                    tell(4u * q + 2u, further);
                }
            }
            else
            {
                const uint32_t acc = labels(dep);
                if (acc == seen)
                    continue;
                seen = acc;
                x = vote(wn, acc, m0, m1);
                if (x == JST_OPEN && local)
                {
                    // the heaviest open neighbour: does it decide alone?
                    float w = -1.0F;
                    uint32_t on = 0u, bit = 0u;
#pragma unroll
                    for (int k = 0; k < 12; ++k)
                        if (((acc >> k) & (acc >> (k + 12)) & 1u) && wn[k] > w)
                        {
                            w = wn[k];
                            on = dep[k];
                            bit = 1u << k;
                        }
                    if (bit != 0u && vote(wn, acc & ~(bit << 12), m0, m1) == V_G && vote(wn, acc & ~bit, m0, m1) == V_O)
                    {
                        copied = on;
                        tell(4u * q + 2u, (on - own) / 4u + 1u);
                    }
                }
            }
            if (x != JST_OPEN)
                decide(q, x);
        }
        if (x != JST_OPEN)
            gst[q] = static_cast<uint8_t>(x);
        else
            leave(at, q);
    }
    __syncwarp();
    cluster_barrier(); // no CTA leaves while another may still write its states
    if (rank == 0u && s_left != 0u)
        vote_rows(RowVote{gst, next, b.jrec + sd.jq_off, b.jq_total, b.row_cnt + sd.row_off, b.row_cols + sd.pix_off,
                          b.pix_depth + sd.pix_off, sd.H, sd.W});
}

// populateLabels (segmenter.cpp:640-669) and the colour image of Segmenter::image().
__device__ __forceinline__ void paint_pixel(uint8_t* image, uint32_t p, uint8_t stv)
{
    uint8_t bgr[3] = {0, 0, 0};
    switch (stv)
    {
    case PX_GROUND:
    case PX_RES_G:
        bgr[1] = 255;
        break;
    case PX_OBSTACLE:
    case PX_RES_O:
    case PX_EMPTY_RED:
        bgr[2] = 255;
        break;
    case PX_INTERSECT:
        bgr[0] = 255;
        break;
    default:
        break;
    }
    image[3 * p] = bgr[0];
    image[3 * p + 1] = bgr[1];
    image[3 * p + 2] = bgr[2];
}

// kPer pixels per thread: four where they fill the SMs, so that their look-ups (the vote's outcome, the label's place)
// run side by side (64 scans: 59 us with one, 33 with four); one where they do not, as the look-ups' latency is
// all there is then (64 x 2048 scan: 6 us with one, 8 with four).
template <uint32_t kPer>
__global__ void k_populate(BatchDev b, uint8_t* image)
{
    pdl_enter();
    const uint32_t p0 = kPer * (blockIdx.x * blockDim.x + threadIdx.x);
    if (p0 >= b.npix)
        return;
    const uint32_t cnt = min(kPer, b.npix - p0);
    uint8_t stv[kPer];
    int32_t li[kPer], all = -1;
    if (kPer == 4u && cnt == 4u)
    {
        const uchar4 a = *reinterpret_cast<const uchar4*>(b.pix_state + p0);
        const int4 m = *reinterpret_cast<const int4*>(b.pix_map + p0);
        const uint8_t as[4] = {a.x, a.y, a.z, a.w};
        const int32_t ms[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u)
        {
            stv[u] = as[u];
            li[u] = ms[u];
        }
    }
    else
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u)
        {
            stv[u] = (u < cnt) ? b.pix_state[p0 + u] : static_cast<uint8_t>(PX_EMPTY);
            li[u] = (u < cnt) ? b.pix_map[p0 + u] : -1;
        }
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u)
        all &= li[u];
    if (all >= 0) // (all -1: no point)
    {
        const int s0 = scan_of_pix(b, p0);
        const bool one = kPer == 1u || s0 + 1 >= b.nscan || p0 + kPer - 1u < b.scans[s0 + 1].pix_off;
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u)
        {
            if (li[u] < 0)
                continue;
            const ScanDev& sd = b.scans[one ? s0 : scan_of_pix(b, p0 + u)];
            if (stv[u] == PX_INTERSECT)
            {
                const uint8_t v = b.jst[sd.jq_off + b.pix_depth[p0 + u]];
                stv[u] = (v == V_O) ? PX_RES_O : ((v == V_G) ? PX_RES_G : PX_INTERSECT);
            }
            const uint8_t v = final_view(stv[u]);
            if (v != V_U)
                b.seg_label[sd.pt_off + static_cast<uint32_t>(li[u])] = (v == V_G) ? LP_LABEL_GROUND : LP_LABEL_OBSTACLE;
        }
    }
    if (image)
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u)
            if (u < cnt)
                paint_pixel(image, p0 + u, stv[u]);
}
} // namespace

// ------------------------------------------------------------------------------------------
// Host launch sequence for the segmentation stage (all launches on one stream, no host sync).
// ------------------------------------------------------------------------------------------
void launch_ring_only(Launcher& L, const BatchDev& b, const BatchHost& hb)
{
    const uint32_t T = 256;
    LP_LAUNCH(L, k_quadrant, div_up(b.npts, T), T, b);
    LP_LAUNCH(L, k_ring_count, hb.ntiles, 256, b);
    L.scan(b.tile_cnt, b.tile_cnt, hb.ntiles + 1);
    LP_LAUNCH(L, k_ring_apply, hb.ntiles, 256, b);
}

__global__ void k_debug_math(int kind, const float* a, const float* bb, uint32_t n, float* out)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    float r;
    switch (kind)
    {
    case 0:
        r = lpm::cr_atan2f(a[i], bb[i]);
        break;
    case 1:
        r = lpm::cr_atanf(a[i]);
        break;
    case 2:
        r = lpm::cr_expf(a[i]);
        break;
    case 4:
        r = lpm::cr_atan2f_fp64(a[i], bb[i]);
        break;
    case 5:
        r = lpm::cr_atanf_fp64(a[i]);
        break;
    case 6:
        r = lpm::cr_expf_fp64(a[i]);
        break;
    default:
        r = lpm::atan2_approx(a[i], bb[i]);
        break;
    }
    out[i] = r;
}

void init_segment_tables()
{
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64 && done[dev])
        return;
    std::mt19937 gen(42u);
    uint32_t table[kMtTable];
    for (int k = 0; k < kMtTable; ++k)
        table[k] = static_cast<uint32_t>(gen());
    const bool attr = cudaFuncSetAttribute(k_jcp_resolve<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           static_cast<int>(4u * kResolveStates + 16u)) == cudaSuccess &&
                      cudaFuncSetAttribute(k_jcp_resolve<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           static_cast<int>(4u * kResolveStates + 16u)) == cudaSuccess;
    if (cudaMemcpyToSymbol(g_mt42, table, sizeof(table)) == cudaSuccess && attr && dev >= 0 && dev < 64)
        done[dev] = true;
}

void launch_debug_math(Launcher& L, int kind, const float* a, const float* bb, uint32_t n, float* out)
{
    LP_LAUNCH(L, k_debug_math, div_up(n, 256u), 256, kind, a, bb, n, out);
}

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z)
{
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// Sweep of the float-float first stage against the binary64 / double-double stages. kind 1
// (atan) and 2 (exp): argument = the float whose bits are `first + i`; kind 0 (atan2): (y, x) from
// a hash of first + i, either arbitrary finite floats or the same with their exponents drawn
// close (ratios near 1, the axes and the diagonals). stats: [0] decided by stage 1, [1] left to
// the later stages, [2] stage 1 decided differently; first_bad: lowest such index.
__global__ void k_debug_math_sweep(int kind, unsigned long long first, unsigned long long count,
                                   unsigned long long* stats, unsigned long long* first_bad)
{
    pdl_enter();
    unsigned long long dec = 0, und = 0, bad = 0;
    const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
    for (unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; i < count;
         i += stride)
    {
        const unsigned long long idx = first + i;
        float f = 0.0f, want = 0.0f;
        bool ok = false;
        if (kind == 1)
        {
            const float x = __uint_as_float(static_cast<uint32_t>(idx));
            ok = lpm::ff_atanf(x, &f);
            if (ok)
                want = lpm::cr_atanf_fp64(x);
        }
        else if (kind == 2)
        {
            const float x = __uint_as_float(static_cast<uint32_t>(idx));
            ok = x >= -87.0f && x <= 88.5f && lpm::ff_expf(x, &f);
            if (ok)
                want = lpm::cr_expf_fp64(x);
        }
        else
        {
            const unsigned long long h = splitmix64(idx);
            uint32_t by = static_cast<uint32_t>(h), bx = static_cast<uint32_t>(h >> 32);
            if (idx & 1ull) // exponents within a few of each other
                bx = (bx & 0x807fffffu) | ((((by >> 23) & 0xffu) + ((bx >> 23) & 7u) - 3u) & 0xffu) << 23;
            if ((idx & 6ull) == 2ull) // ties of magnitude: the diagonals
                bx = (bx & 0x80000000u) | (by & 0x7fffffffu);
            const float y = __uint_as_float(by), x = __uint_as_float(bx);
            ok = lpm::ff_atan2f(y, x, &f);
            if (ok)
                want = lpm::cr_atan2f_fp64(y, x);
        }
        if (!ok)
            ++und;
        else
        {
            ++dec;
            if (__float_as_uint(f) != __float_as_uint(want))
            {
                ++bad;
                atomicMin(first_bad, idx);
            }
        }
    }
    dec = __reduce_add_sync(0xffffffffu, static_cast<uint32_t>(dec));
    und = __reduce_add_sync(0xffffffffu, static_cast<uint32_t>(und));
    bad = __reduce_add_sync(0xffffffffu, static_cast<uint32_t>(bad));
    if (lane_id() == 0)
    {
        atomicAdd(&stats[0], dec);
        atomicAdd(&stats[1], und);
        atomicAdd(&stats[2], bad);
    }
}

void launch_debug_math_sweep(Launcher& L, int kind, unsigned long long first, unsigned long long count,
                             unsigned long long* stats, unsigned long long* first_bad)
{
    LP_LAUNCH(L, k_debug_math_sweep, 152u * 16u, 256, kind, first, count, stats, first_bad);
}

void launch_segmentation(Launcher& L, const BatchDev& b, const BatchHost& hb, uint8_t* d_image)
{
    const uint32_t T = 256;
    if (hb.any_compute_ring)
        launch_ring_only(L, b, hb);
    LP_LAUNCH(L, k_bin, div_up(b.npts, 2u * T), T, b);
    L.scan(b.cell_cnt, b.cell_start, b.ncell + 1);
    LP_LAUNCH(L, k_scatter, div_up(b.npts, T), T, b);
    if (b.npts / 16u < hb.nslices)
        LP_LAUNCH(L, k_recm_sparse, div_up(hb.nslices, kRecmThreads / 32u), kRecmThreads, b, hb.nslices);
    else
        LP_LAUNCH(L, k_recm, hb.nslices, kRecmThreads, b);
    LP_LAUNCH(L, k_ransac_draw, static_cast<uint32_t>(b.nscan) * kDrawCtas, kDrawThreads, b);
    // about four CTAs per SM over the batch's tiles
    // (candidates are points: more CTAs than their tiles would only take tickets)
    const uint32_t most = static_cast<uint32_t>(sm_count()) * 4u;
    const uint32_t each = b.npts < most * kInlierTile ? kInlierTileFew : kInlierTile;
    L.launch("k_ransac_inliers", each == kInlierTile ? k_ransac_inliers<kInlierTile> : k_ransac_inliers<kInlierTileFew>,
             std::min(most, b.npts / each + static_cast<uint32_t>(b.nscan)), 256, b);
    const bool many = b.npix > static_cast<uint32_t>(sm_count()) * 10240u; // four pixels per thread fill the SMs
    const uint32_t pix_ctas = div_up(b.npix, many ? 4u * T : T);
    if (hb.packed_key)
    {
        L.launch("k_label_depth", k_label_depth<true>, div_up(b.npts, T), T, b);
        L.launch("k_pixel", many ? k_pixel<true, 4> : k_pixel<true, 1>, pix_ctas, T, b);
    }
    else
    {
        L.launch("k_label_depth", k_label_depth<false>, div_up(b.npts, T), T, b);
        LP_LAUNCH(L, k_project_key, div_up(b.npts, T), T, b);
        L.launch("k_pixel", many ? k_pixel<false, 4> : k_pixel<false, 1>, pix_ctas, T, b);
    }
    LP_LAUNCH(L, k_dilate_rows, b.nrows, 256, b);
    LP_LAUNCH(L, k_jcp_weights, static_cast<uint32_t>(sm_count()) * hb.jcp_ctas_per_sm, kWeightThreads, b);
    uint32_t cap = 16u; // the queue holds at most the scan's pixels and points
    for (const ScanDev& sd : hb.scans)
        cap = std::max(cap, std::min((sd.jq_cap + 15u) & ~15u, kResolveStates));
    const uint32_t ns = static_cast<uint32_t>(b.nscan);
    if (b.nscan <= kResolveWide)
        L.launch_smem("k_jcp_resolve", k_jcp_resolve<8>, ns * 8u, kResolveThreads, 4u * cap + 16u, b, cap);
    else
        L.launch_smem("k_jcp_resolve", k_jcp_resolve<4>, ns * 4u, kResolveThreads, 4u * cap + 16u, b, cap);
    L.launch("k_populate", many ? k_populate<4> : k_populate<1>, pix_ctas, T, b, d_image);
}
} // namespace lpg
