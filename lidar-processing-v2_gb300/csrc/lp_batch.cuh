// lp_batch.cuh — device pointers of one batch (passed by value to every kernel).
//
// HBM layout: each array is flat over the batch; scan s owns [ScanDev::*_off, + count).
//   points       float4 xyzi (16 B)            npts      (after optional noise compaction)
//   pixels       state u8, map i32, keys u64    npix      = sum H*W
//   polar cells  counts/starts/elevation        ncell     = sum nslice*nrad
//   near cells   RANSAC candidate counts        nnear     = sum nslice*4
//   obstacles    float4 + src index             <= npts
//   voxel hash   key/min/count                  nhash     = sum pow2 >= 2*n
//   clusters     counts/starts/boxes            ncl       = sum (n/min_size + 1)
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "lp_internal.cuh"

namespace lpg
{
// Pixel states of the range image (the reference's BGR colours, segmenter.hpp:144-148).
enum : uint8_t
{
    PX_EMPTY = 0,     // (0,0,0)
    PX_GROUND = 1,    // (0,255,0)
    PX_OBSTACLE = 2,  // (0,0,255)
    PX_INTERSECT = 4, // (255,0,0)   queued, not (yet) resolved by the vote
    PX_EMPTY_RED = 6, // (0,0,255)   empty pixel whose red channel was dilated
    PX_RES_G = 7,     // (0,255,0)   queued pixel the vote resolved to ground
    PX_RES_O = 8      // (0,0,255)   queued pixel the vote resolved to obstacle
};

// Vote outcomes / labels seen by a neighbour: 0 unknown, 1 ground, 2 obstacle.
enum : uint8_t
{
    V_U = 0,
    V_G = 1,
    V_O = 2
};

constexpr uint32_t kKtPoolPerPoint = 8; // leftover search entries per point the DROR pool holds
// Raw weight record of the jump convolution: 24 weights, padded to a multiple of 16 bytes.
constexpr uint32_t kJwStride = 28;
constexpr uint32_t kNearCopies = 4; // one per CTA that draws a scan's hypotheses
constexpr uint32_t kJrecFields = 10; // 16-byte fields of an open pixel's record (jrec in lp_segment.cu)

// A scan's buffers in the caller's page-locked host memory (device-accessible addresses).
struct IoScan
{
    const float* xyzi;
    const uint16_t* ring;
    uint8_t* noise;
    uint32_t* seg;
    int32_t* cl;
    uint32_t* hoff;
    int32_t* hidx;
    float* zmin;
    float* zmax;
    lp_bounding_box* obbc;
    lp_bounding_box* obbp;
    uint32_t cluster_cap, hull_cap;
    uint32_t q_off; // first label tile of the scan in the batch's tile list
};
constexpr uint32_t kIoTile = 1024; // points per label tile

// Offsets of scans 1..7 in the batch arrays (0xffffffff past the last), in the kernels' arguments: up to
// eight scans (a part of a split batch) are told apart by seven comparisons against constant operands;
// the search of the descriptors costs a chain of three to six loads per thread of every kernel.
constexpr int kFewScans = 8;
struct FewOffsets
{
    uint32_t at[kFewScans - 1];
    __device__ __forceinline__ int find(uint32_t i) const
    {
        int s = 0;
#pragma unroll
        for (int k = 0; k < kFewScans - 1; ++k)
            s += (i >= at[k]) ? 1 : 0;
        return s;
    }
};

struct BatchDev
{
    int nscan;
    FewOffsets pt_few, pix_few, row_few, slice_few, cl_few;
    const ScanDev* scans;
    ScanState* state;

    // ---- input / points --------------------------------------------------------------------
    uint32_t nsrc;            // input points (before noise compaction)
    const float4* src;        // input points
    uint8_t* noise;           // per input point: LP_NOISE_*
    uint32_t* src_pos;        // per input point: compacted position (scan of VALID flags)
    uint32_t npts;            // points entering segmentation
    float4* pts;              // compacted points (== src when noise removal is off)
    int32_t* pt_src;          // compacted point -> input point (global)
    uint16_t* ring;           // per compacted point
    const uint16_t* ring_in;  // per input point, or null
    IoScan* io;               // per scan: the caller's page-locked buffers (direct host I/O)

    // ---- ring partition ---------------------------------------------------------------------
    uint8_t* quad;            // per point quadrant
    uint32_t ntiles;
    uint32_t* tile_cnt;       // transitions per 1024-point tile -> exclusive scan in place

    // ---- polar grid --------------------------------------------------------------------------
    int32_t* pt_cell;  // global cell or -1
    int32_t* pt_pix;   // local pixel h*W+w
    uint32_t* pt_slot; // arrival slot in the cell
    uint32_t ncell;
    uint32_t* cell_cnt;
    uint32_t* cell_start;
    int32_t* csr_idx;  // local point index per grid entry
    float* csr_z;
    float* zlow;       // per cell
    float* elev;       // per cell
    uint32_t* large_list; // per slice (at its first cell): cells whose heights have to be sorted

    // ---- RANSAC ------------------------------------------------------------------------------
    uint32_t nnear;
    uint32_t* near_cnt;   // RANSAC candidates per near cell
    uint32_t* near_start; // kNearCopies x nnear: first candidate rank of each near cell
    float4* cand;         // candidates of a scan from its pt_off, unordered
    float4* planes;            // nscan * 60
    unsigned long long* pvalid; // nscan: bit it = hypothesis it usable
    uint32_t* inliers;         // nscan * 60
    uint32_t* ransac_done;     // CTAs of the inlier count that have finished

    // ---- projection / range image ------------------------------------------------------------
    uint8_t* pt_label; // per point after RECM + RANSAC
    uint32_t npix;
    uint32_t* pix_depth;
    unsigned long long* pix_key;
    int32_t* pix_map;
    uint8_t* pix_state;

    // ---- jump convolution -------------------------------------------------------------------
    uint32_t nrows;
    uint16_t* row_cols;        // per pixel slot: intersection columns of the row in order
    uint4* jq;            // per scan (jq_off): its queued pixels: (image row, position | column << 16, point, 0)
    uint32_t* row_cnt;         // per global row
    float* jw;                 // per row, its last three queued pixels: 24 fresh weights (stride kJwStride)
    uint32_t jq_total;         // queue capacity: sum over scans of min(pixels, points), each rounded up to 16
    uint8_t* jst;              // per queued pixel: its outcome, or JST_OPEN
    uint4* jrec;               // per open pixel (list position at jq_off): kJrecFields x jq_total
    uint32_t* jlist;           // 2 x jq_total: positions of the pixels still open, round by round
    uint32_t* jborder;         // list positions of the open pixels whose window leaves the image

    // ---- segmentation output -----------------------------------------------------------------
    uint32_t* seg_label; // per compacted point

    // ---- clustering --------------------------------------------------------------------------
    uint32_t* obs_flag;   // per point: 1 if obstacle -> exclusive scan in place (obstacle slot)
    float4* obs_pts;      // per obstacle: x, y, z, (float)local index
    int32_t* obs_pt;      // per obstacle: compacted point index (global)
    float* obs_r;
    float* obs_a;
    float* obs_e;
    uint32_t* obs_hslot;  // per obstacle: hash slot
    uint32_t nhash;
    uint4* hrec;          // voxel hash: key (0xffffffff: free), smallest local obstacle, points, union-find parent slot
    uint32_t* vlist;      // hash slots of the batch's voxels
    uint32_t* kflag;      // per obstacle: kept components whose smallest obstacle lies before it
    int32_t* obs_label;   // per obstacle: cluster label or -1

    // ---- per-cluster ---------------------------------------------------------------------------
    uint32_t ncl;
    uint32_t hull_cta_min; // clusters of more members take a CTA of the hull kernel (tuning)
    uint32_t* cl_cnt;     // members per cluster
    uint32_t* cl_start;   // first member slot of each cluster (disjoint ranges, in the order of cl_rank)
    uint32_t* cl_rank;
    uint32_t* cl_fill;
    uint32_t* members;    // obstacle indices grouped by cluster (unordered within)
    float2* mxy;          // x, y of each member, by member slot
    uint32_t* cl_zkey;    // per cluster: max of ~ord(z) (the lowest z), max of ord(z) (the highest)
    uint32_t* hull_cnt;   // hull vertices per cluster -> per scan, offsets into hull_out (from its pt_off)
    int32_t* hull_tmp;    // per member slot: hull local indices at cl_start
    int32_t* hull_out;    // dense hull local indices (batch)
    float* cl_zmin;
    float* cl_zmax;
    lp_bounding_box* obb_c;
    lp_bounding_box* obb_p;
    void* hs_cand;        // hull candidates (12 B each), 2 per member slot, at 2 * cl_start
    int32_t* hs_stack;    // monotone-chain stack, at 2 * cl_start + 2 * cl_rank
    double2* hs_pts;      // hull vertices as FP64, at cl_start
    int2* hs_pairs;       // antipodal pairs, at 4 * cl_start + 16 * cl_rank
    uint32_t* hull_work;  // hull work list: large clusters from the front, the others from the back
    uint32_t* queue;      // [8..9] member slots and clusters given a range, [1] large-cluster head, [2] large clusters, [3] others,
                          // [4] others' head, [5] tie clusters, [6] chunks of the member passes
    uint32_t* tie_list;
    uint2* pre_items;          // (cluster, chunk) items of the large clusters' member passes
    unsigned long long* pre_ext;  // per cluster: its 16 direction extremes (packed keys)
    unsigned long long* pre_pk;   // per cluster: the farthest member outside each edge of the first polygon
    uint32_t* pre_nact;        // per cluster: members not inside the first polygon (listed in the chain scratch)   // clusters whose hull has a vertex with an identical point (reference tie order)

    // ---- DROR (reference kd-tree replay, lp_kdtree.cu) ------------------------------------------
    float4* kt;                // per input point: tree node record by position (x, y, z, subtree size bits)
    float4* kbb;               // 2 per input point: subtree box (lo, hi) by node position
    uint32_t* kscr;            // 2 per input point: candidate positions of the parallel partition (later,
                               // per candidate: its walk through its predecessor's stop pieces: stop entry, left at)
    uint32_t* kown;            // per point: count of its own search (capped at min_neighbours); later, per
                               // candidate: the count after that walk
    uint32_t* kshort;          // per point (+1): 1 if its own search fell short -> exclusive scan
    uint32_t* klo_n;           // per point (+1): entries its search left behind; later, per short point:
                               // the first flat entry of its piece
    uint32_t* klo_off;         // exclusive scan of klo_n: their place in kflat
    uint32_t* klo_at;          // per point: their place in kpool; later, per candidate: that walk's status,
                               // left count and stop piece
    uint32_t* kpool;           // leftover entries as searches produce them (kpool_cap)
    uint32_t* kflat;           // the points' leftovers in point order (kpool_cap)
    uint32_t kpool_cap;
    uint32_t* kq;              // short points in order (before that, from the build to the own search:
                               // the input index of the point at each tree position)
    uint4* kc;                 // per short point: count, stop entry, left entries (pool at, count)
    uint32_t* kcflag;          // per short point (+1): 1 if step 3 left it undecided -> exclusive scan
    uint32_t* kcand;           // those candidates (short indices) in order
    uint4* kspec;              // per candidate: count, stop short index, stop entry | kind << 31, left at; later,
                               // at a run's first candidate: its result (k_kt_run)
    uint32_t* kspec_n;         // per candidate: entries the stopping search left
    uint2* kpiece;             // per scan: stacks of pieces (2 n + 2 per scan)
    uint32_t* kctr;            // [0] pool head, [1] stopped candidates
    uint32_t* kstop;           // stopped candidates in order (klo_off, no longer read by then)

    // ---- outputs per input point ---------------------------------------------------------------
    uint32_t* out_seg;
    int32_t* out_cl;
};

__device__ __forceinline__ int scan_of_point(const BatchDev& b, uint32_t i)
{
    return b.nscan <= kFewScans ? b.pt_few.find(i) : find_scan(b.nscan, i, [&](int s) { return b.scans[s].pt_off; });
}
__device__ __forceinline__ int scan_of_cluster(const BatchDev& b, uint32_t g)
{
    return b.nscan <= kFewScans ? b.cl_few.find(g) : find_scan(b.nscan, g, [&](int s) { return b.scans[s].cl_off; });
}
} // namespace lpg
