// lp_internal.cuh — batch layout shared by the kernels of liblp_gpu.so.
//
// A batch is S scans laid out back to back in device memory (HBM). Every per-point, per-pixel,
// per-cell array of the batch is one flat array; a scan owns the slice [off, off + count) of
// each, recorded in its ScanDev descriptor. A single scan is a batch of one, so the plain
// (one scan per launch sequence) and the batched form run the same kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "lidar_gb300.h"

namespace lpg
{
constexpr int kMaxRansacIters = 60;  // segmenter.cpp:324
constexpr int kRansacRadialBins = 4; // segmenter.cpp:323
constexpr uint32_t kVoxelCapacity = 200000u; // clusterer.cpp:36 (StaticUnorderedMap reserve)

// Error bits raised by kernels in ScanState::err (read back with the results).
enum : uint32_t
{
    ERR_CELL_TOO_LARGE = 1u << 0,
    ERR_VOXEL_CAPACITY = 1u << 1,
    ERR_HASH_FULL = 1u << 2,
    ERR_HULL_CAPACITY = 1u << 3,
    ERR_CLUSTER_CAPACITY = 1u << 4,
    ERR_UF_TIMEOUT = 1u << 5,
    ERR_INTERNAL = 1u << 6,
};

// Static per-scan description: sizes, offsets into the batch arrays and configuration values
// precomputed on the host with the same binary32 expressions the reference evaluates.
struct ScanDev
{
    // points (after optional noise compaction)
    uint32_t pt_off, n;
    uint32_t src_off, n_src; // original input points (before noise compaction)
    // range image
    uint32_t pix_off;
    int32_t H, W;
    uint32_t row_off;   // first global row (sum of H of earlier scans)
    uint32_t jq_off, jq_cap; // vote queue slice: jq_off a multiple of 16, at most min(pixels, points) entries
    uint32_t tile_off;  // first 1024-point ring tile
    uint32_t slice_off; // first global azimuth slice
    // polar grid
    uint32_t cell_off;
    int32_t nslice, nrad;
    uint32_t near_off; // near-field cells (radial < 4), nslice * min(4, nrad)
    int32_t nnear_per_slice;
    // segmentation constants (segmenter.cpp:106-122, :209-211, :360)
    float zmin_adj, zmax_adj, spacing, min_d, max_d, slice_res;
    float down_rad, rad_per_px;
    float delta, thr, sensor_h, kthr2, amp, max_cos;
    // projection key (project_key): bits of the least squared distance, shifts of distance and cell
    uint32_t key_base, key_dist, key_cell;
    int32_t use_ring; // 1: height index from ring; 0: from the elevation angle
    int32_t compute_ring;
    int32_t first_ring;
    // clustering constants (clusterer.hpp:76-90)
    float res_r, res_a, res_e;
    uint32_t min_cluster;
    uint32_t hash_cap; // most voxel hash slots the scan can need (power of two)
    // per-cluster output capacity
    uint32_t cluster_cap, hull_cap;
    uint32_t cl_off; // offset of this scan's cluster arrays
    uint32_t hull_off;
    // DROR (noise_remover.cpp:49-57): s2 = pow(double(multiplier), 2), rmin2 = rmin * rmin
    double dror_s2;
    float dror_rmin2;
    uint32_t dror_k;
};

// Dynamic per-scan values produced on the device.
struct ScanState
{
    uint32_t err;
    uint32_t n_pts;     // points entering segmentation (after noise removal)
    // RANSAC (segmenter.cpp:321-479)
    uint32_t n_cand, cand_off;
    int32_t ransac_ok;
    float plane[4];
    // clustering
    uint32_t n_obs, obs_off;
    uint32_t max_r_bits, max_a_bits, max_e_bits;
    int32_t nr, na, ne;
    uint32_t hash_off, hash_mask; // voxel hash slice: first slot, slots - 1
    uint32_t n_vox;
    uint32_t n_comp; // of the batch's first scan: voxels listed (all scans)
    uint32_t n_clusters;
    // jump convolution: queued pixels, those the weights pass left open, and of these the ones whose
    // window leaves the image
    uint32_t n_queue, n_open, n_border;
    uint32_t pad[7]; // to a line of 128 bytes: scans' counters do not share one
};
static_assert(sizeof(ScanState) == 128);

// First statement of every kernel. Launches of a run carry the programmatic-serialisation attribute
// (Launcher), so a kernel's CTAs may be set up while the one before it drains: it waits here until that
// one is complete and its writes are visible, then lets its own successor be set up. A no-op in other
// launches.
__device__ __forceinline__ void pdl_enter()
{
    asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void raise_err(ScanState* st, uint32_t bit)
{
    atomicOr(&st->err, bit);
}

// Binary search of the scan that owns flat index `i` given ascending offsets.
template <typename F>
__device__ __forceinline__ int find_scan(int nscan, uint32_t i, F off_of)
{
    int lo = 0, hi = nscan - 1;
    while (lo < hi)
    {
        const int mid = (lo + hi + 1) >> 1;
        if (off_of(mid) <= i)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ uint32_t lane_id()
{
    return threadIdx.x & 31u;
}

// Elements per tile of a device-wide scan over n elements. A tile is one CTA: short scans take small
// tiles, so that their loads spread over the chip (1,024 elements up to 1 Mi: at most 1,024 tiles to
// look back over), long ones large tiles, so that the look-back stays short.
__host__ __device__ constexpr uint32_t scan_tile(uint32_t n)
{
    return n <= (1u << 20) ? 1024u : 8192u;
}
// 64-bit words a scan over n elements needs (zeroed): the ticket counter and one per tile.
__host__ __device__ constexpr uint32_t scan_words(uint32_t n)
{
    return (n + scan_tile(n) - 1u) / scan_tile(n) + 1u;
}

// At least scan_words(m) for every m <= n (short scans have small tiles, so they can need more).
__host__ __device__ constexpr uint32_t scan_words_max(uint32_t n)
{
    return scan_words(n) > scan_words(1u << 20) ? scan_words(n) : scan_words(n < (1u << 20) ? n : 1u << 20);
}

} // namespace lpg
