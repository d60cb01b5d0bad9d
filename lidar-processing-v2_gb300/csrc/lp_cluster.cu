// lp_cluster.cu — curved-voxel clustering of the obstacle points.
//
// Reference: lidar_processing_lib/src/clusterer.cpp. The reference labels 26-connected
// components of occupied (range, azimuth, elevation) voxels by a BFS seeded in point order, so
// a component's label is the rank of its smallest point index; components smaller than
// min_cluster_size are dropped and the rest renumbered in the same order (clusterer.cpp:
// 122-239). Here: a per-scan open-addressing hash of occupied voxels, lock-free union-find over
// the 26-neighbour graph (the azimuth index wraps modulo num_azimuth as in clusterer.cpp:
// 161-169), and the canonical labels from a prefix scan of "component minimum" flags. Labels
// are identical to the reference's, not only the partition.
#include <algorithm>

#include "lp_batch.cuh"
#include "lp_common.cuh"
#include "lp_math.cuh"
#include "lp_stages.hpp"

namespace lpg
{
namespace
{
constexpr float kTwoPiF = 6.28318548202514648438f; // Clusterer::TWO_M_PIf
constexpr float kPi2F = 1.57079637050628662109f;   // M_PI_2f
constexpr uint32_t kEmpty = 0xffffffffu;
constexpr int kMaxIters = 1 << 22;

__device__ __forceinline__ int scan_of_obs(const BatchDev& b, uint32_t o)
{
    return b.nscan == 1 ? 0 : find_scan(b.nscan, o, [&](int s) { return b.state[s].obs_off; });
}
__device__ __forceinline__ int scan_of_hash(const BatchDev& b, uint32_t h)
{
    return b.nscan == 1 ? 0 : find_scan(b.nscan, h, [&](int s) { return b.state[s].hash_off; });
}
__device__ __forceinline__ uint32_t hash_mix(uint32_t k)
{
    k *= 0x9E3779B1u;
    k ^= k >> 15;
    k *= 0x85EBCA77u;
    k ^= k >> 13;
    return k;
}
__device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p)
{
    return *reinterpret_cast<const volatile uint32_t*>(p);
}

// Obstacle slots: the exclusive scan of "is an obstacle" over the points.
struct ObsFlagSrc
{
    const uint32_t* label;
    uint32_t n;
    __device__ __forceinline__ uint32_t end() const { return 0xffffffffu; }
    __device__ __forceinline__ uint4 get4(uint32_t i) const
    {
        uint4 v = ScanSrcU32{label, n, true}.get4(i); // (no label is LP_LABEL_OBSTACLE past the end)
        return make_uint4(v.x == LP_LABEL_OBSTACLE, v.y == LP_LABEL_OBSTACLE, v.z == LP_LABEL_OBSTACLE, v.w == LP_LABEL_OBSTACLE);
    }
};

// The scans' obstacle ranges and voxel hash slices, by the first warp of a block (every lane returns the
// slots of all scans together). The slice of a scan holds next_pow2(max(64, 2 n_obs)) slots, packed
// one scan after the other: sized by the obstacles, not by the points, the hash of a 64 x 2048 scan
// is 16 to 64 times smaller (its clearing and every pass over it with it) and stays in L2.
__device__ __forceinline__ uint32_t hash_layout(const BatchDev& b, bool write)
{
    uint32_t base = 0u;
    for (int s0 = 0; s0 < b.nscan; s0 += 32)
    {
        const int s = s0 + static_cast<int>(lane_id());
        uint32_t slots = 0u, off = 0u, n = 0u;
        if (s < b.nscan)
        {
            const ScanDev& sd = b.scans[s];
            off = b.obs_flag[sd.pt_off];
            n = b.obs_flag[sd.pt_off + sd.n] - off;
            slots = next_pow2(max(64u, 2u * n)); // <= hash_cap: n <= sd.n
        }
        const uint32_t incl = warp_incl_scan(slots);
        if (write && s < b.nscan)
        {
            ScanState& st = b.state[s];
            st.obs_off = off;
            st.n_obs = n;
            st.hash_off = base + incl - slots;
            st.hash_mask = slots - 1u;
        }
        base += __shfl_sync(0xffffffffu, incl, 31);
    }
    return base;
}

// Obstacle cloud in input order (processor.cpp:562-579) with the spherical coordinates of
// Clusterer::cartesianToSpherical (clusterer.cpp:55-100). A block takes 1024 consecutive points
// and first compacts its obstacle points in shared memory, so that every lane of the arithmetic
// below (two correctly rounded arctangents) has one. The grid also clears the voxel hash, and its first
// block records the scans' obstacle ranges and hash slices.
constexpr uint32_t kObsChunk = 1024;

__global__ void __launch_bounds__(256) k_obs_gather(BatchDev b)
{
    pdl_enter();
    __shared__ uint32_t sidx[kObsChunk];
    __shared__ uint32_t scnt, s_slots;
    const uint32_t base = blockIdx.x * kObsChunk;
    if (threadIdx.x < 32u)
    {
        const uint32_t slots = hash_layout(b, blockIdx.x == 0u);
        if (threadIdx.x == 0)
        {
            scnt = 0u;
            s_slots = slots;
        }
    }
    __syncthreads();
    for (uint32_t h = blockIdx.x * 256u + threadIdx.x; h < s_slots; h += gridDim.x * 256u)
        b.hrec[h] = make_uint4(kEmpty, kEmpty, 0u, h);
#pragma unroll
    for (uint32_t u = 0; u < kObsChunk / 256u; ++u)
    {
        const uint32_t i = base + u * 256u + threadIdx.x;
        const bool valid = i < b.npts && b.seg_label[i] == LP_LABEL_OBSTACLE;
        const uint32_t m = __ballot_sync(0xffffffffu, valid);
        uint32_t pos = 0u;
        if (lane_id() == 0 && m)
            pos = atomicAdd(&scnt, static_cast<uint32_t>(__popc(m)));
        pos = __shfl_sync(0xffffffffu, pos, 0);
        if (valid)
            sidx[pos + static_cast<uint32_t>(__popc(m & ((1u << lane_id()) - 1u)))] = i;
    }
    __syncthreads();
    const uint32_t cnt = scnt;
    for (uint32_t k0 = 0; k0 < cnt; k0 += 256u)
    {
        const uint32_t k = k0 + threadIdx.x;
        const bool valid = k < cnt;
        const uint32_t i = valid ? sidx[k] : 0u;
        const int s = valid ? scan_of_point(b, i) : -1;
        uint32_t rb = 0u, ab = 0u, eb = 0u;
        if (valid)
        {
            const uint32_t o = b.obs_flag[i];
            const float4 p = b.pts[i];
            b.obs_pts[o] = p;
            b.obs_pt[o] = static_cast<int32_t>(i);
            float az = lpm::cr_atan2f(p.y, p.x);
            az = (az < 0) ? (az + kTwoPiF) : az;
            const float d2 = p.x * p.x + p.y * p.y;
            const float d = sqrtf(d2);
            const float r = sqrtf(d2 + p.z * p.z);
            const float el = lpm::cr_atanf(p.z / d) + kPi2F;
            b.obs_r[o] = r;
            b.obs_a[o] = az;
            b.obs_e[o] = el;
            rb = r > 0.0f ? __float_as_uint(r) : 0u; // non-negative floats order like their bits
            ab = az > 0.0f ? __float_as_uint(az) : 0u;
            eb = el > 0.0f ? __float_as_uint(el) : 0u;
        }
        // one atomic per warp when the warp's obstacle points belong to a single scan
        const int smax = static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<unsigned>(s + 1))) - 1;
        if (__all_sync(0xffffffffu, s == smax || s < 0))
        {
            rb = __reduce_max_sync(0xffffffffu, rb);
            ab = __reduce_max_sync(0xffffffffu, ab);
            eb = __reduce_max_sync(0xffffffffu, eb);
            if (lane_id() == 0 && smax >= 0)
            {
                ScanState& st = b.state[smax];
                atomicMax(&st.max_r_bits, rb);
                atomicMax(&st.max_a_bits, ab);
                atomicMax(&st.max_e_bits, eb);
            }
        }
        else if (valid)
        {
            ScanState& st = b.state[s];
            atomicMax(&st.max_r_bits, rb);
            atomicMax(&st.max_a_bits, ab);
            atomicMax(&st.max_e_bits, eb);
        }
    }
}

__device__ __forceinline__ int32_t flat_voxel(int32_t nr, int32_t na, int32_t r, int32_t a, int32_t e)
{
    return nr * (na * e + a) + r; // Clusterer::flatVoxelIndex, clusterer.hpp:136-142
}

// Voxel hash slot (hrec): key, smallest obstacle of the voxel, its point count, union-find parent (a
// slot; itself until linked). One 16-byte record, so an insertion and a lookup touch one sector each.
// New voxels are listed (vlist; state[0].n_comp counts the batch's). The grid dimensions
// (clusterer.cpp:92-99) come from the maxima that k_obs_gather left; the thread of a scan's first
// obstacle records them.
// What bounds it is the L2's atomics: neighbours in a row share their voxel and every new voxel its scan's
// counters, so the lanes of a warp that fell into one voxel insert it once, and a CTA takes its place in the list
// and counts its voxels with one atomic each (obstacle by obstacle and warp by warp, 64 scans took 92 us).
constexpr uint32_t kVoxThreads = 256;
__global__ void __launch_bounds__(kVoxThreads) k_vox_insert(BatchDev b)
{
    pdl_enter();
    __shared__ uint32_t wnew[kVoxThreads / 32], wbase[kVoxThreads / 32];
    __shared__ int ends[2]; // the scans of the CTA's first and last obstacle
    const uint32_t nobs = b.obs_flag[b.npts];
    const uint32_t o0 = blockIdx.x * kVoxThreads;
    if (o0 >= nobs)
        return;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t o = o0 + threadIdx.x;
    const bool in = o < nobs;
    const int s = scan_of_obs(b, min(o, nobs - 1u));
    const ScanDev& sd = b.scans[s];
    ScanState& st = b.state[s];
    const int32_t nr = static_cast<int32_t>(ceilf(__uint_as_float(st.max_r_bits) / sd.res_r) + 1.0f);
    const int32_t na = static_cast<int32_t>(ceilf(__uint_as_float(st.max_a_bits) / sd.res_a) + 1.0f);
    uint32_t key = 0u;
    if (in)
    {
        if (o == st.obs_off)
        {
            const int32_t ne = static_cast<int32_t>(ceilf(__uint_as_float(st.max_e_bits) / sd.res_e) + 1.0f);
            st.nr = nr;
            st.na = na;
            st.ne = ne;
            if (static_cast<long long>(nr) * na * ne > 0x7fffffffLL)
                raise_err(&st, ERR_INTERNAL);
        }
        const int32_t vr = static_cast<int32_t>(b.obs_r[o] / sd.res_r);
        const int32_t va = static_cast<int32_t>(b.obs_a[o] / sd.res_a);
        const int32_t ve = static_cast<int32_t>(b.obs_e[o] / sd.res_e);
        key = static_cast<uint32_t>(flat_voxel(nr, na, vr, va, ve));
    }
    const unsigned long long voxel = in ? (static_cast<unsigned long long>(s) << 32) | key : ~0ull;
    const uint32_t peers = __match_any_sync(0xffffffffu, voxel);
    const int leader = __ffs(peers) - 1; // the smallest obstacle of the warp's in the voxel
    bool fresh = false;
    uint32_t at = kEmpty;
    if (in && static_cast<int>(lane) == leader)
    {
        const uint32_t mask = st.hash_mask, off = st.hash_off;
        uint32_t h = hash_mix(key) & mask;
        for (uint32_t probe = 0; probe <= mask; ++probe)
        {
            uint32_t* rec = reinterpret_cast<uint32_t*>(&b.hrec[off + h]);
            const uint32_t prev = atomicCAS(&rec[0], kEmpty, key);
            if (prev == kEmpty || prev == key)
            {
                at = off + h;
                fresh = prev == kEmpty;
                atomicMin(&rec[1], o - st.obs_off);
                atomicAdd(&rec[2], static_cast<uint32_t>(__popc(peers)));
                break;
            }
            h = (h + 1u) & mask;
        }
        if (at == kEmpty)
            raise_err(&st, ERR_HASH_FULL);
    }
    at = __shfl_sync(0xffffffffu, at, leader);
    if (in)
        b.obs_hslot[o] = at;
    const uint32_t m = __ballot_sync(0xffffffffu, fresh);
    if (lane == 0)
        wnew[warp] = static_cast<uint32_t>(__popc(m));
    if (threadIdx.x == 0 || threadIdx.x == kVoxThreads - 1u)
        ends[threadIdx.x != 0] = s;
    __syncthreads();
    if (warp == 0)
    {
        const uint32_t v = (lane < kVoxThreads / 32u) ? wnew[lane] : 0u;
        const uint32_t incl = warp_incl_scan(v);
        uint32_t base = 0u;
        if (lane == 31u && incl)
        {
            base = atomicAdd(&b.state[0].n_comp, incl);
            if (ends[0] == ends[1]) // (the obstacles lie scan by scan)
                atomicAdd(&st.n_vox, incl);
        }
        base = __shfl_sync(0xffffffffu, base, 31);
        if (lane < kVoxThreads / 32u)
            wbase[lane] = base + incl - v;
    }
    __syncthreads();
    if (!fresh)
        return;
    b.vlist[wbase[warp] + static_cast<uint32_t>(__popc(m & ((1u << lane) - 1u)))] = at;
    if (ends[0] != ends[1])
        atomicAdd(&st.n_vox, 1u);
}

// Every parent pointer is strictly smaller than its index except at roots (links go from the
// larger root to the smaller; path halving only shortens), so a find ends within x steps. The
// per-thread budget bounds the total work anyway: exhausting it raises ERR_UF_TIMEOUT.
__device__ __forceinline__ uint32_t* parent_of(uint4* rec, uint32_t x)
{
    return &rec[x].w;
}

__device__ uint32_t uf_find(uint4* rec, uint32_t x, ScanState* st, int& budget)
{
    while (budget-- > 0)
    {
        const uint32_t p = ld_volatile(parent_of(rec, x));
        if (p == x)
            return x;
        const uint32_t gp = ld_volatile(parent_of(rec, p));
        if (gp != p)
            atomicCAS(parent_of(rec, x), p, gp); // path halving; parents only ever decrease
        x = gp;
    }
    raise_err(st, ERR_UF_TIMEOUT);
    return x;
}

__device__ void uf_union(uint4* rec, uint32_t a, uint32_t c, ScanState* st, int& budget)
{
    while (budget > 0)
    {
        a = uf_find(rec, a, st, budget);
        c = uf_find(rec, c, st, budget);
        if (budget <= 0)
            return;
        if (a == c)
            return;
        if (a > c)
        {
            const uint32_t t = a;
            a = c;
            c = t;
        }
        // link the larger root below the smaller one
        const uint32_t old = atomicCAS(parent_of(rec, c), c, a);
        if (old == c)
            return;
        c = old;
    }
    raise_err(st, ERR_UF_TIMEOUT);
}

__device__ __forceinline__ uint32_t hash_lookup(const BatchDev& b, const ScanState& st, uint32_t key)
{
    const uint32_t mask = st.hash_mask, off = st.hash_off;
    uint32_t h = hash_mix(key) & mask;
    for (uint32_t probe = 0; probe <= mask; ++probe)
    {
        const uint32_t k = b.hrec[off + h].x;
        if (k == key)
            return off + h;
        if (k == kEmpty)
            return kEmpty;
        h = (h + 1u) & mask;
    }
    return kEmpty;
}

// Neighbour offsets (clusterer.hpp:101-105): all 26 (dr, da, de) != (0, 0, 0). Only the 13 after
// (0, 0, 0) in (de, da, dr) order are probed: every adjacent pair of voxels is then met from one
// side (or both, where the azimuth wraps onto itself), which yields the same components as probing
// all 26. One (voxel, offset) pair per thread: the probes are chains of dependent loads, so they
// run side by side; the components (and the labels, component minima) do not depend on the order
// of the unions.
__device__ __forceinline__ void k_uf_hook_pair(const BatchDev& b, uint32_t v, uint32_t o)
{
    // offset o: 0 -> (de 0, da 0, dr +1), 1..3 -> (0, +1, -1..+1), 4..12 -> (+1, -1..+1, -1..+1)
    const int32_t de = (o < 4u) ? 0 : 1;
    const int32_t da = (o == 0u) ? 0 : ((o < 4u) ? 1 : static_cast<int32_t>((o - 4u) / 3u) - 1);
    const int32_t dr = (o == 0u) ? 1 : ((o < 4u) ? static_cast<int32_t>(o) - 2 : static_cast<int32_t>((o - 4u) % 3u) - 1);
    const uint32_t slot = b.vlist[v];
    ScanState* st = &b.state[scan_of_hash(b, slot)];
    const int32_t nr = st->nr, na = st->na, ne = st->ne;
    const int32_t key = static_cast<int32_t>(b.hrec[slot].x);
    const int32_t r = key % nr;
    const int32_t a = (key / nr) % na;
    const int32_t e = key / (nr * na);
    const int32_t rr = r + dr, ee = e + de;
    if (rr < 0 || rr >= nr || ee < 0 || ee >= ne)
        return;
    int32_t aa = a + da;
    if (aa < 0)
        aa += na;
    else if (aa >= na)
        aa -= na;
    const uint32_t nslot = hash_lookup(b, *st, static_cast<uint32_t>(flat_voxel(nr, na, rr, aa, ee)));
    if (nslot != kEmpty && nslot != slot)
    {
        int budget = kMaxIters;
        uf_union(b.hrec, slot, nslot, st, budget);
    }
}

// The union-find runs on the hash slots themselves: their order is random, so neighbouring voxels'
// roots do not contend, and no pass has to number the voxels.
__global__ void k_uf_hook(BatchDev b)
{
    pdl_enter();
    if (blockIdx.x == 0)
        for (int s = static_cast<int>(threadIdx.x); s < b.nscan; s += static_cast<int>(blockDim.x))
            if (b.state[s].n_vox > kVoxelCapacity)
                raise_err(&b.state[s], ERR_VOXEL_CAPACITY); // StaticUnorderedMap::insert throws (static_unordered_map.hpp:81)
    const uint32_t nv = b.state[0].n_comp; // voxels; threads stride over (offset, voxel) pairs
    const unsigned long long total = 13ull * nv;
    for (unsigned long long t = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; t < total;
         t += static_cast<unsigned long long>(gridDim.x) * blockDim.x)
        k_uf_hook_pair(b, static_cast<uint32_t>(t % nv), static_cast<uint32_t>(t / nv));
}

// Every voxel straight below its root, and the components' smallest obstacle and point count in the
// root's record (its own are the start; the other voxels' records keep theirs).
__global__ void k_uf_flatten(BatchDev b)
{
    pdl_enter();
    const uint32_t nv = b.state[0].n_comp;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x)
    {
        const uint32_t slot = b.vlist[v];
        int budget = kMaxIters;
        const uint32_t root = uf_find(b.hrec, slot, &b.state[scan_of_hash(b, slot)], budget);
        if (root == slot)
            continue;
        uint4* rec = &b.hrec[slot];
        rec->w = root;
        uint32_t* rr = reinterpret_cast<uint32_t*>(&b.hrec[root]);
        atomicMin(&rr[1], rec->y);
        atomicAdd(&rr[2], rec->z);
    }
}

// Component flags in obstacle order: 1 at the smallest obstacle of every component that is kept
// (removeSmallClusters, clusterer.cpp:195-239). The obstacle's root is left in obs_label for the pass
// after the scan.
struct KeepSrc
{
    BatchDev b;
    __device__ __forceinline__ uint32_t end() const { return b.obs_flag[b.npts] + 1u; }
    __device__ __forceinline__ uint32_t one(uint32_t o, uint32_t n) const
    {
        if (o >= n)
            return 0u;
        const uint32_t slot = b.obs_hslot[o];
        if (slot == kEmpty)
        {
            b.obs_label[o] = -1;
            return 0u;
        }
        const uint32_t root = b.hrec[slot].w;
        b.obs_label[o] = static_cast<int32_t>(root);
        const int s = scan_of_obs(b, o);
        const uint4 r = b.hrec[root];
        return (r.y == o - b.state[s].obs_off && r.z >= b.scans[s].min_cluster) ? 1u : 0u;
    }
    __device__ __forceinline__ uint4 get4(uint32_t i) const
    {
        const uint32_t n = b.obs_flag[b.npts];
        return make_uint4(one(i, n), one(i + 1u, n), one(i + 2u, n), one(i + 3u, n));
    }
};

// kflag now holds the exclusive scan: rank of each kept component among the scan's kept
// components ordered by smallest point index == the reference's final label.
__global__ void k_obs_label(BatchDev b)
{
    pdl_enter();
    __shared__ BlockAgg agg;
    if (blockIdx.x == 0)
        for (int s = static_cast<int>(threadIdx.x); s < b.nscan; s += static_cast<int>(blockDim.x))
        {
            ScanState& st = b.state[s];
            st.n_clusters = b.kflag[st.obs_off + st.n_obs] - b.kflag[st.obs_off];
            if (st.n_clusters > b.scans[s].cluster_cap)
                raise_err(&st, ERR_CLUSTER_CAPACITY);
        }
    const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = o < b.obs_flag[b.npts];
    int32_t label = LP_INVALID_CLUSTER;
    uint32_t g = 0u;
    if (in)
    {
        const int s = scan_of_obs(b, o);
        const ScanDev& sd = b.scans[s];
        const ScanState& st = b.state[s];
        const int32_t root = b.obs_label[o]; // a hash slot (KeepSrc)
        if (root >= 0)
        {
            const uint4 r = b.hrec[root];
            if (r.z >= sd.min_cluster)
                label = static_cast<int32_t>(b.kflag[st.obs_off + r.y] - b.kflag[st.obs_off]);
        }
        b.obs_label[o] = label;
        g = sd.cl_off + static_cast<uint32_t>(label);
    }
    block_aggregated_inc(b.cl_cnt, g, in && label >= 0, agg);
}

// Members grouped by cluster (slot order within a cluster is free), with their x, y alongside for
// the hull stage, and each cluster's z range (ordered-key maxima: one atomic pair per cluster and
// warp where a warp's points share few clusters; otherwise per point, skipped when a fresh read
// of the key shows it cannot rise).
__device__ __forceinline__ uint32_t z_ord(float f)
{
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__global__ void k_cl_scatter(BatchDev b)
{
    pdl_enter();
    __shared__ BlockAgg agg;
    const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = lane_id();
    const int32_t label = (o < b.obs_flag[b.npts]) ? b.obs_label[o] : -1;
    const bool in = label >= 0;
    uint32_t g = 0u;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    if (in)
    {
        g = b.scans[scan_of_obs(b, o)].cl_off + static_cast<uint32_t>(label);
        p = b.obs_pts[o];
    }
    const uint32_t rank = block_aggregated_inc(b.cl_fill, g, in, agg);
    if (in)
    {
        const uint32_t slot = b.cl_start[g] + rank;
        b.members[slot] = o;
        b.mxy[slot] = make_float2(p.x, p.y);
    }
    const uint32_t zo = z_ord(p.z);
    const uint32_t peers = __match_any_sync(0xffffffffu, in ? g : 0xffffffffu);
    const uint32_t groups = __popc(__ballot_sync(0xffffffffu, in && lane == static_cast<uint32_t>(__ffs(peers) - 1)));
    if (groups > 4u)
    {
        if (in)
        {
            if (~zo > __ldcg(&b.cl_zkey[2u * g]))
                atomicMax(&b.cl_zkey[2u * g], ~zo);
            if (zo > __ldcg(&b.cl_zkey[2u * g + 1u]))
                atomicMax(&b.cl_zkey[2u * g + 1u], zo);
        }
        return;
    }
    for (uint32_t todo = __ballot_sync(0xffffffffu, in); todo != 0u;)
    {
        const int l = __ffs(todo) - 1;
        const uint32_t lg = __shfl_sync(0xffffffffu, g, l);
        const bool mine = in && g == lg;
        const uint32_t lo = __reduce_max_sync(0xffffffffu, mine ? ~zo : 0u);
        const uint32_t hi = __reduce_max_sync(0xffffffffu, mine ? zo : 0u);
        if (lane == static_cast<uint32_t>(l))
        {
            atomicMax(&b.cl_zkey[2u * lg], lo);
            atomicMax(&b.cl_zkey[2u * lg + 1u], hi);
        }
        todo &= ~__ballot_sync(0xffffffffu, mine);
    }
}
} // namespace

// Clusterer::cluster on a caller-supplied cloud: every point is a member of the cloud to cluster.
__global__ void k_mark_all(BatchDev b)
{
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.npts)
        return;
    const int s = scan_of_point(b, i);
    b.seg_label[i] = (i - b.scans[s].pt_off < b.state[s].n_pts) ? LP_LABEL_OBSTACLE : LP_LABEL_UNKNOWN;
}

void launch_mark_all_obstacles(Launcher& L, const BatchDev& b)
{
    LP_LAUNCH(L, k_mark_all, div_up(b.npts, 256u), 256, b);
}

void launch_clustering(Launcher& L, const BatchDev& b, const BatchHost& hb)
{
    (void)hb;
    const uint32_t T = 256;
    auto scan = [&](const char* name, auto src, uint32_t* out) {
        if (uint32_t* words = L.scan_state(b.npts + 1))
        {
            L.begin(name);
            scan_lookback(L.stream, src, ScanDstU32{out, b.npts + 1, true}, b.npts + 1, words, L.scan_err, true, L.overlap);
            L.end();
            L.note();
        }
    };
    scan("k_obs_scan", ObsFlagSrc{b.seg_label, b.npts}, b.obs_flag);
    LP_LAUNCH(L, k_obs_gather, div_up(b.npts, kObsChunk), 256, b);
    LP_LAUNCH(L, k_vox_insert, div_up(b.npts, kVoxThreads), kVoxThreads, b);
    const uint32_t vgrid = std::min(div_up(13u * std::max(b.npts, 1u), T), static_cast<uint32_t>(sm_count()) * 8u);
    LP_LAUNCH(L, k_uf_hook, vgrid, T, b);
    LP_LAUNCH(L, k_uf_flatten, std::min(div_up(b.npts, T), static_cast<uint32_t>(sm_count()) * 8u), T, b);
    scan("k_keep_scan", KeepSrc{b}, b.kflag);
    LP_LAUNCH(L, k_obs_label, div_up(b.npts, T), T, b);
}

void launch_cluster_scatter(Launcher& L, const BatchDev& b)
{
    LP_LAUNCH(L, k_cl_scatter, div_up(b.npts, 256u), 256, b);
}
} // namespace lpg
