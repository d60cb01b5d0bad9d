// lp_io.cu — scan inputs read and results written directly in the caller's page-locked host
// buffers, over the GPU's coherent host link (NVLink-C2C on GB300), one kernel each way instead of
// one copy per array per scan. Used by lp_process_batch when every buffer of the call was
// allocated with lp_host_alloc.
#include <algorithm>

#include "lp_batch.cuh"
#include "lp_common.cuh"
#include "lp_stages.hpp"

namespace lpg
{
namespace
{
// Input points (and rings) of every scan into the batch arrays. A small grid-strided grid (two
// CTAs per SM) with four host loads in flight per thread: the host link's rate needs far fewer
// threads than one per point, and the other parts of a split batch keep the remaining SMs for
// their compute while this part's inputs stream in.
__global__ void k_io_in(BatchDev b, const IoScan* io)
{
    pdl_enter();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < b.nsrc; i0 += 4u * stride)
    {
        float4 v[4];
        uint16_t rg[4] = {0, 0, 0, 0};
        uint32_t at[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const uint32_t i = i0 + static_cast<uint32_t>(u) * stride;
            at[u] = 0xffffffffu;
            if (i >= b.nsrc)
                continue;
            const int s = scan_of_point(b, i); // (src_off == pt_off)
            const ScanDev& sd = b.scans[s];
            const uint32_t k = i - sd.src_off;
            if (k >= sd.n_src)
                continue;
            const IoScan& d = io[s];
            v[u] = reinterpret_cast<const float4*>(d.xyzi)[k];
            if (b.ring_in && d.ring)
                rg[u] = d.ring[k];
            at[u] = i;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (at[u] != 0xffffffffu)
            {
                const_cast<float4*>(b.src)[at[u]] = v[u];
                if (b.ring_in)
                    const_cast<uint16_t*>(b.ring_in)[at[u]] = rg[u];
            }
    }
}

// Results into the caller's page-locked buffers, one launch. What bounds it is the host link, which
// takes 190 GB/s of whole 128-byte lines from as few as 38 CTAs and 80 GB/s or less of lines that a
// warp's store fills in part (measured with 16-byte stores 32 bytes apart). The buffers of a batch
// are usually slices of one array, at any offset, so no store may count on the alignment of its
// point number: a tile's labels are gathered in shared memory and written with lanes on consecutive words
// of the destination, each warp on one of its lines, whatever the offset. (One thread per four points
// with 16-byte stores, or four 4-byte stores where the offset was odd, ran at 64 GB/s: 32 scans of a
// batch 600 us; the 64-scan call 3.23 -> 2.41 ms, six scans 620 -> 578 us, with this kernel.)
constexpr int kIoThreads = 256;
constexpr uint32_t kIoClusterCtas = 8; // CTAs per scan for its clusters' results

struct IoSmem
{
    uint32_t seg[kIoTile];
    int32_t cl[kIoTile];
    uint8_t nz[kIoTile];
};

// n words to dst, lane by lane along dst's 128-byte lines.
template <class T>
__device__ __forceinline__ void put_lines(T* dst, const T* from, uint32_t n)
{
    static_assert(sizeof(T) == 4);
    const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(dst) >> 2) & 31u;
    for (uint32_t i = threadIdx.x; i < n + lead; i += kIoThreads)
        if (i >= lead)
            dst[i - lead] = from[i - lead];
}

// n bytes to dst: whole words along its lines, bytes at the ends.
__device__ __forceinline__ void put_lines(uint8_t* dst, const uint8_t* from, uint32_t n)
{
    const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(dst)) & 127u;
    for (uint32_t w = 4u * threadIdx.x; w < n + lead; w += 4u * kIoThreads)
    {
        if (w >= lead && w + 4u <= n + lead)
        {
            const uint8_t* f = from + (w - lead);
            *reinterpret_cast<uint32_t*>(dst + (w - lead)) = static_cast<uint32_t>(f[0]) | (static_cast<uint32_t>(f[1]) << 8) |
                                                             (static_cast<uint32_t>(f[2]) << 16) |
                                                             (static_cast<uint32_t>(f[3]) << 24);
            continue;
        }
        for (uint32_t u = max(w, lead); u < min(w + 4u, n + lead); ++u)
            dst[u - lead] = from[u - lead];
    }
}

// Per-point labels, tile q of the batch (scan s with io[s].q_off <= q, its points kIoTile (q - q_off) ..),
// straight from the stages' arrays (by compacted point, by obstacle), without a pass of their own.
__device__ __forceinline__ void io_out_tile(const BatchDev& b, const IoScan* io, IoSmem& sm, uint32_t q)
{
    const int s = find_scan(b.nscan, q, [&](int t) { return io[t].q_off; });
    const ScanDev& sd = b.scans[s];
    const IoScan& d = io[s];
    const uint32_t k0 = kIoTile * (q - d.q_off);
    if (k0 >= sd.n_src) // (a scan without points has no tile)
        return;
    const uint32_t i0 = sd.src_off + k0;
    const uint32_t cnt = min(kIoTile, sd.n_src - k0);
    const bool filtered = b.pt_src != nullptr;
    const uint32_t src0 = filtered ? b.src_pos[sd.src_off] : 0u;
#pragma unroll
    for (uint32_t u = 0; u < kIoTile / kIoThreads; ++u)
    {
        const uint32_t t = u * kIoThreads + threadIdx.x;
        if (t < cnt)
        {
            uint32_t pos = i0 + t; // compacted point
            uint8_t nz = 0;
            uint32_t sg = 0;
            int32_t cl = LP_INVALID_CLUSTER;
            if (filtered)
            {
                nz = b.noise[i0 + t];
                pos = sd.pt_off + (b.src_pos[i0 + t] - src0);
            }
            if (!filtered || nz == LP_NOISE_VALID)
            {
                sg = b.seg_label[pos];
                if (d.cl && sg == LP_LABEL_OBSTACLE)
                    cl = b.obs_label[b.obs_flag[pos]];
            }
            sm.nz[t] = nz;
            sm.seg[t] = sg;
            sm.cl[t] = cl;
        }
    }
    __syncthreads();
    if (d.noise)
        put_lines(d.noise + k0, sm.nz, cnt);
    if (d.seg)
        put_lines(d.seg + k0, sm.seg, cnt);
    if (d.cl)
        put_lines(d.cl + k0, sm.cl, cnt);
    __syncthreads(); // (the tile is read before the next one is gathered)
}

// n words to dst, CTA `part` of kIoClusterCtas.
__device__ __forceinline__ void put_part(void* dst, const void* from, uint32_t n, uint32_t part)
{
    for (uint32_t i = part * kIoThreads + threadIdx.x; i < n; i += kIoClusterCtas * kIoThreads)
        static_cast<uint32_t*>(dst)[i] = static_cast<const uint32_t*>(from)[i];
}

// Per-cluster results of scan s: hull offsets (relative to the scan), hull indices, z range, boxes, each a
// contiguous range on both sides. A scan whose clusters or hull indices exceed the caller's capacities
// gets none of them (the host reports LP_ERR_CAPACITY for it). ret[s] = the scan's hull index count
// (page-locked host memory).
__device__ __forceinline__ void io_out_clusters(const BatchDev& b, const IoScan* io, uint32_t* ret, int with_obb, int s,
                                                uint32_t part)
{
    const ScanDev& sd = b.scans[s];
    const IoScan& d = io[s];
    const uint32_t kcl = b.state[s].n_clusters;
    const uint32_t* off = b.hull_cnt + sd.cl_off;
    const uint32_t base = off[0];
    const uint32_t nh = kcl < sd.cluster_cap ? off[kcl] - base : 0u;
    if (part == 0 && threadIdx.x == 0)
        ret[s] = nh;
    if (kcl >= sd.cluster_cap || kcl > d.cluster_cap || nh > d.hull_cap)
        return;
    if (d.hoff)
        for (uint32_t k = part * kIoThreads + threadIdx.x; k <= kcl; k += kIoClusterCtas * kIoThreads)
            d.hoff[k] = off[k] - base;
    if (d.hidx)
        put_part(d.hidx, b.hull_out + base, nh, part);
    if (d.zmin)
        put_part(d.zmin, b.cl_zmin + sd.cl_off, kcl, part);
    if (d.zmax)
        put_part(d.zmax, b.cl_zmax + sd.cl_off, kcl, part);
    static_assert(sizeof(lp_bounding_box) % 4 == 0);
    if (with_obb && d.obbc)
        put_part(d.obbc, b.obb_c + sd.cl_off, kcl * static_cast<uint32_t>(sizeof(lp_bounding_box) / 4), part);
    if (with_obb && d.obbp)
        put_part(d.obbp, b.obb_p + sd.cl_off, kcl * static_cast<uint32_t>(sizeof(lp_bounding_box) / 4), part);
}

// CTAs [0, ncluster): kIoClusterCtas per scan, its clusters; the others the nq label tiles. host_state: the
// scans' states as the host reads them (page-locked).
__global__ void __launch_bounds__(kIoThreads) k_io_out(BatchDev b, const IoScan* io, uint32_t* ret, ScanState* host_state,
                                                       int with_obb, uint32_t ncluster, uint32_t nq)
{
    __shared__ IoSmem sm;
    pdl_enter();
    if (blockIdx.x < ncluster)
    {
        io_out_clusters(b, io, ret, with_obb, static_cast<int>(blockIdx.x / kIoClusterCtas), blockIdx.x % kIoClusterCtas);
        return;
    }
    const uint32_t first = blockIdx.x - ncluster;
    if (first == 0)
        for (uint32_t i = threadIdx.x; i < static_cast<uint32_t>(b.nscan) * (sizeof(ScanState) / 4u); i += kIoThreads)
            reinterpret_cast<uint32_t*>(host_state)[i] = reinterpret_cast<const uint32_t*>(b.state)[i];
    for (uint32_t q = first; q < nq; q += gridDim.x - ncluster)
        io_out_tile(b, io, sm, q);
}
} // namespace

void launch_io_in(Launcher& L, const BatchDev& b, const IoScan* io)
{
    LP_LAUNCH(L, k_io_in, std::min(div_up(b.nsrc, 256u), static_cast<uint32_t>(sm_count()) * 2u), 256, b, io);
}

void launch_io_out(Launcher& L, const BatchDev& b, const IoScan* io, uint32_t* ret, ScanState* host_state, int with_hull,
                   int with_obb, uint32_t nq)
{
    const uint32_t ncluster = with_hull ? static_cast<uint32_t>(b.nscan) * kIoClusterCtas : 0u;
    const uint32_t tiles = std::min(std::max(nq, 1u), static_cast<uint32_t>(sm_count()) * 2u);
    LP_LAUNCH(L, k_io_out, ncluster + tiles, kIoThreads, b, io, ret, host_state, with_obb, ncluster, nq);
}
} // namespace lpg
