// lp_common.cu — device-wide exclusive scan of u32 arrays (the look-back kernel is in lp_common.cuh).
#include <algorithm>
#include <cstddef>

#include "lp_common.cuh"
#include "lp_stages.hpp"

namespace lpg
{
// Exclusive scan of n u32 (in place allowed). `sums` is the scan scratch (at least
// 8 * scan_words(n) bytes, 8-byte aligned; `zeroed`: already zero), `err` the error word (or null).
void scan_exclusive(cudaStream_t st, const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* sums, uint32_t* err,
                    uint64_t& launches, bool zeroed, bool overlap)
{
    const bool vec = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0u;
    scan_lookback(st, ScanSrcU32{in, n, vec}, ScanDstU32{out, n, vec}, n, sums, err, zeroed, overlap);
    launches += 1;
}

namespace
{
// A wait that nothing will satisfy, to check that bounded waits give up and report: an mbarrier
// expecting one arrival that never comes, polled `limit` times.
__global__ void k_debug_mbar_timeout(uint32_t limit, uint32_t* err)
{
    pdl_enter();
    __shared__ unsigned long long bar;
    if (threadIdx.x == 0)
        mbar_init(&bar, 1u);
    __syncthreads();
    if (!mbar_wait(&bar, 0u, limit) && threadIdx.x == 0)
        atomicOr(err, static_cast<uint32_t>(ERR_INTERNAL));
}
} // namespace

// kind 0: a look-back scan over one tile whose ticket counter starts at 1, so its only block takes
// tile 1 and waits for tile 0's word, which no block writes (every element lies past n: nothing is
// read or written besides the state words); kind 1: an mbarrier wait without an arrival. Both give
// up after `limit` polls and set ERR_INTERNAL in *err. `state` holds at least 4 words.
void launch_debug_wait_timeout(cudaStream_t st, int kind, uint32_t limit, unsigned long long* state, uint32_t* err,
                               uint64_t& launches)
{
    if (kind == 0)
    {
        const unsigned long long start[4] = {1ull, 0ull, 0ull, 0ull};
        cudaMemcpyAsync(state, start, sizeof(start), cudaMemcpyHostToDevice, st);
        k_scan_lb<8><<<1, kLbThreads, 0, st>>>(ScanSrcU32{nullptr, 0u, false}, ScanDstU32{nullptr, 0u, false}, state, err,
                                            limit);
    }
    else
    {
        k_debug_mbar_timeout<<<1, 32, 0, st>>>(limit, err);
    }
    launches += 1;
}
// ------------------------------------------------------------------------------------------
// Everything a run starts from (zeroed counters, empty keys, look-back words, the scans' states) in one
// launch: the ranges are the kernel's argument. As one memset per array (29 of them) they were more than
// a third of a single scan's stream operations, about 3 us of host time and 2 us of device time each
// (graph replay of a 64 x 2048 scan 0.381 -> 0.312 ms with this and the labels written to the host straight
// from the stages' arrays).
// ------------------------------------------------------------------------------------------
namespace
{
__global__ void __launch_bounds__(256) k_prepare(FillList f, BatchDev b, int noise)
{
    pdl_enter();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (int q = 0; q < f.n; ++q)
    {
        const FillRange r = f.r[q];
        const uint4 v = make_uint4(r.value, r.value, r.value, r.value);
        uint4* p = static_cast<uint4*>(r.p);
        for (uint32_t i = t; i < r.n16; i += step)
            p[i] = v;
    }
    constexpr uint32_t kWords = sizeof(ScanState) / 4u, kPts = offsetof(ScanState, n_pts) / 4u;
    for (uint32_t i = t; i < static_cast<uint32_t>(b.nscan) * kWords; i += step)
        reinterpret_cast<uint32_t*>(b.state)[i] = (i % kWords == kPts && !noise) ? b.scans[i / kWords].n : 0u;
}
} // namespace

void launch_prepare(Launcher& L, const FillList& f, const BatchDev& b, int noise)
{
    uint32_t units = 1u;
    for (int q = 0; q < f.n; ++q)
        units = std::max(units, f.r[q].n16);
    LP_LAUNCH(L, k_prepare, std::min(div_up(units, 256u), static_cast<uint32_t>(sm_count()) * 8u), 256, f, b, noise);
}
} // namespace lpg
