// lp_stages.hpp — host-side launch helpers and the stage entry points of liblp_gpu.so.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include <string>
#include <vector>

#include "lp_batch.cuh"

namespace lpg
{
void scan_exclusive(cudaStream_t st, const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* sums, uint32_t* err,
                    uint64_t& launches, bool zeroed = false, bool overlap = false);
void launch_debug_wait_timeout(cudaStream_t st, int kind, uint32_t limit, unsigned long long* state, uint32_t* err,
                               uint64_t& launches);

// Ranges a run starts from (k_prepare): 16-byte units of a 32-bit pattern. Every array of a batch is
// 256-byte aligned with 16 bytes after its end, so a range may be rounded up to whole units.
struct FillRange
{
    void* p;
    uint32_t n16, value;
};
struct FillList
{
    FillRange r[24];
    int n = 0;
    void add(void* p, size_t bytes, uint32_t value)
    {
        r[n++] = FillRange{p, static_cast<uint32_t>((bytes + 15) / 16), value};
    }
};
// Device-wide scans of one run at most (ring tiles, outlier filter 4 + compaction, cells, near cells,
// obstacles, voxels, components, clusters, hulls): each takes its own zeroed look-back words.
constexpr uint32_t kScansPerRun = 13;

// One timed launch (profiling mode only).
struct LaunchRecord
{
    const char* name;
    cudaEvent_t start, stop;
};

// A launch; overlap: its CTAs may be set up while the kernel before it on the stream drains (pdl_enter).
template <typename... P, typename... Args>
void launch_kernel(bool overlap, cudaStream_t stream, void (*kernel)(P...), dim3 grid, uint32_t block, size_t smem, Args... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Issues kernel launches on one stream, counts them and remembers the first launch error. In
// profiling mode every launch is bracketed by CUDA events on the same stream.
struct Launcher
{
    cudaStream_t stream = nullptr;
    uint64_t* launches = nullptr;
    uint32_t* scan_sums = nullptr; // next zeroed look-back words (k_prepare zeroes scan_left of them)
    size_t scan_left = 0;          // 8-byte words left
    uint32_t* scan_err = nullptr;  // error word the device-wide scans report into
    // Launches overlap their predecessor's end where the run has the stream's SMs to itself (graph replay
    // of a 64 x 2048 scan 0.238 -> 0.228 ms). Not in the parts of a split batch: the other parts fill
    // those gaps already, and CTAs that wait hold their SMs (64 scans in eight parts: 1.73 -> 1.85 ms).
    bool overlap = false;
    cudaError_t err = cudaSuccess;
    std::vector<LaunchRecord>* prof = nullptr;
    std::vector<cudaEvent_t>* event_pool = nullptr;
    size_t pool_next = 0;

    cudaEvent_t next_event()
    {
        if (pool_next >= event_pool->size())
        {
            cudaEvent_t e;
            cudaEventCreate(&e);
            event_pool->push_back(e);
        }
        return (*event_pool)[pool_next++];
    }
    void begin(const char* name)
    {
        if (prof)
        {
            LaunchRecord r{name, next_event(), next_event()};
            cudaEventRecord(r.start, stream);
            prof->push_back(r);
        }
    }
    void end()
    {
        if (prof)
            cudaEventRecord(prof->back().stop, stream);
    }

    template <typename K, typename... Args>
    void issue(K kernel, dim3 grid, uint32_t block, size_t smem, Args... args)
    {
        launch_kernel(overlap, stream, kernel, grid, block, smem, args...);
    }
    template <typename K, typename... Args>
    void launch(const char* name, K kernel, uint32_t grid, uint32_t block, Args... args)
    {
        if (grid == 0 || err != cudaSuccess)
            return; // nothing runs after a failed step: its inputs would be undefined
        begin(name);
        issue(kernel, dim3(grid), block, 0, args...);
        end();
        note();
    }
    template <typename K, typename... Args>
    void launch_smem(const char* name, K kernel, uint32_t grid, uint32_t block, size_t smem, Args... args)
    {
        if (grid == 0 || err != cudaSuccess)
            return; // nothing runs after a failed step: its inputs would be undefined
        begin(name);
        issue(kernel, dim3(grid), block, smem, args...);
        end();
        note();
    }
    void scan(const uint32_t* in, uint32_t* out, uint32_t n)
    {
        if (n == 0)
            return;
        uint32_t* words = scan_state(n);
        if (!words)
            return;
        begin("k_scan");
        scan_exclusive(stream, in, out, n, words, scan_err, *launches, true, overlap);
        end();
        note_only();
    }
    // Look-back words of a scan over n elements (null, with the error noted, when the run has none left).
    uint32_t* scan_state(uint32_t n)
    {
        const size_t words = scan_words(n);
        if (words > scan_left || err != cudaSuccess)
        {
            if (err == cudaSuccess)
                err = cudaErrorInvalidValue;
            return nullptr;
        }
        uint32_t* p = scan_sums;
        scan_sums += 2u * words;
        scan_left -= words;
        return p;
    }
    void note()
    {
        ++(*launches);
        note_only();
    }
    void note_only()
    {
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess && err == cudaSuccess)
            err = e;
    }
};

#define LP_LAUNCH(L, k, grid, block, ...) (L).launch(#k, k, grid, block, __VA_ARGS__)
#define LP_LAUNCH_SMEM(L, k, grid, block, smem, ...) (L).launch_smem(#k, k, grid, block, smem, __VA_ARGS__)

// One-time kernel attributes (dynamic shared memory opt-in); called when a context is created.
void init_kernel_attributes();
void init_kdtree_attributes(); // lp_kdtree.cu
// Direct host I/O (lp_io.cu): inputs from and results into the caller's page-locked buffers.
void launch_io_in(Launcher& L, const BatchDev& b, const IoScan* io);
void launch_io_out(Launcher& L, const BatchDev& b, const IoScan* io, uint32_t* ret, ScanState* host_state, int with_hull,
                   int with_obb, uint32_t nq);
void init_segment_tables(); // per-device constant tables (the seed-42 MT19937 stream)
// PointCloud2 bytes -> XYZI (+ ring) (lp_wire.cu); offsets: x, y, z, intensity, ring.
void launch_unpack_pointcloud2(cudaStream_t st, const uint8_t* data, uint32_t width, uint32_t height,
                               uint32_t point_step, uint32_t row_step, const uint32_t* offsets, float4* xyzi,
                               uint16_t* ring, uint64_t& launches);
// The processor's ground / obstacle / unsegmented clouds (lp_split.cu): out holds 3 x n records.
void launch_split_clouds(cudaStream_t st, const float4* pts, const uint32_t* labels, uint32_t n, lp_xyzrgb* out,
                         uint32_t* counts, uint32_t* sums, uint64_t& launches);
// Per-cluster products after the hulls (lp_objects.cu, k_obj_gate in lp_hull.cu).
struct RandWindow // glibc rand()'s last 34 values; pos: the slot the next value replaces
{
    uint32_t r[34];
    uint32_t pos;
};
struct VehicleTableDev // processor.hpp:60-192 in binary64: min/max length, width, height; bounds
{
    double dims[5][6];
    double bounds[5][4]; // min/max volume, min/max area
    double min_h, max_h, min_v, max_v;
};
struct ObjDev
{
    uint32_t K;
    const uint32_t* cl_off;   // K + 1: first cloud slot of each cluster
    const uint32_t* hull_off; // K + 1
    const int32_t* hull_idx;  // local indices
    const float* zmin;
    const float* zmax;
    int32_t* cls;             // K: vehicle type or -1
    lp_bounding_box* boxes;   // K: the gate's calipers boxes
    const lp_xyzrgb* cloud;   // the clustered cloud
    uint32_t* moff;           // K + 1: marker points per cluster -> exclusive scan
    double* mpts;             // marker points (3 doubles each)
    uint32_t mcap;
};
uint32_t obj_tiles(uint32_t n);
void launch_objects_cloud(cudaStream_t st, const float4* pts, const int32_t* labels, uint32_t n, uint32_t K,
                          uint32_t* cnt, uint32_t* sums, uint32_t* err, const RandWindow& w, uchar4* colour,
                          uint32_t* cl_off, lp_xyzrgb* cloud, uint64_t& launches);
void launch_objects_gates(cudaStream_t st, const ObjDev& o, const VehicleTableDev& vt, int enabled, double2* P,
                          float2* Pf, float* ea, int2* pairs, ScanState* state, uint64_t& launches);
void launch_objects_markers(cudaStream_t st, const ObjDev& o, uint32_t* sums, uint64_t& launches);

// Streaming multiprocessors of the current device (persistent grids are sized by it).
int sm_count();

// Host-side sizes of a batch (what the kernels' grids are sized by).
struct BatchHost
{
    int nscan = 0;
    bool any_compute_ring = false;
    bool packed_key = true; // every scan's projection keys fit one word (k_label_depth)
    uint32_t ntiles = 0;
    uint32_t nslices = 0;
    std::vector<ScanDev> scans;
    // launch shapes (lp_tuning)
    uint32_t hull_ctas_per_sm = 2;
    uint32_t jcp_ctas_per_sm = 8;
};

void launch_segmentation(Launcher& L, const BatchDev& b, const BatchHost& hb, uint8_t* d_image);
void launch_ring_only(Launcher& L, const BatchDev& b, const BatchHost& hb);
void launch_clustering(Launcher& L, const BatchDev& b, const BatchHost& hb);
void launch_cluster_scatter(Launcher& L, const BatchDev& b); // members by cluster, for the hulls
void launch_polygons(Launcher& L, const BatchDev& b, const BatchHost& hb, int compute_obb);
void launch_noise(Launcher& L, const BatchDev& b, const BatchHost& hb, const lp_noise_remover_config& cfg);
void launch_noise_compaction(Launcher& L, const BatchDev& b, const BatchHost& hb);
void launch_prepare(Launcher& L, const FillList& f, const BatchDev& b, int noise);
void launch_outputs(Launcher& L, const BatchDev& b, int with_clusters);
void launch_mark_all_obstacles(Launcher& L, const BatchDev& b);
void launch_hull_single(Launcher& L, const double2* pts, uint32_t n, void* scratch, int* stack, int32_t* out,
                        uint32_t* n_out);
void launch_boxes_single(Launcher& L, const double2* P, uint32_t n, int2* pairs, int cap, int kind,
                         lp_bounding_box* out, int* npairs_out);
void launch_debug_math(Launcher& L, int kind, const float* a, const float* b, uint32_t n, float* out);
void launch_debug_math_sweep(Launcher& L, int kind, unsigned long long first, unsigned long long count,
                             unsigned long long* stats, unsigned long long* first_bad);
} // namespace lpg
