/*
 * ryoanji-b200: kernels of the batched solve (many independent systems, one launch per phase).
 *
 * The systems are concatenated: system s owns the bodies [first[s], first[s + 1]). Each body's key is its system
 * index in the top 3L bits (L = sysLevel octree levels) followed by the top 63 - 3L bits of its Hilbert key in the
 * system's own box. Sorting these keys sorts every system along its own curve and keeps the systems in place; the
 * cornerstone tree over them holds each system's tree below the level-L node of its prefix (leaves holding bodies
 * are forced to level >= L so no leaf spans two systems). A system's tree equals its stand-alone tree wherever
 * the stand-alone tree stops above level 21 - L.
 *
 * The reference solves one system per call (ryoanji/test/demo.cu:82-104); there is no batched counterpart.
 */
#include <cstddef>

#include "internal.hpp"

namespace ryo
{

//! system of body i: the last s with first[s] <= i
__device__ __forceinline__ uint32_t systemOf(const uint64_t* __restrict__ first, uint32_t numSystems, uint64_t i)
{
    uint32_t lo = 0, hi = numSystems - 1;
    while (lo < hi)
    {
        uint32_t mid = (lo + hi + 1) >> 1;
        if (__ldg(first + mid) <= i) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

constexpr int kRangeStep = 8 * kWarp; // bodies per round of a warp

/*! per-system minima and maxima of kArrays arrays, as ordered bits: (min, max) of each array from @p out + s *
 *  @p stride on, which hold the neutral values at the start. A warp has @p chunk consecutive bodies and adds its result
 *  of every system among them with one atomic per value. With kSkipNaN NaNs are passed over, as by fminf and fmaxf.
 *  Bound by the latency of its loads and atomics. 2.7M bodies in 256 systems: coordinates 15 us, softenings and masses
 *  10 us. With 64 bodies in a row per thread, whose loads are not coalesced, the coordinates took 62 us; with a block
 *  per system, which waits for the largest, the softenings and masses 69 us. */
template<int kArrays, bool kSkipNaN>
__global__ void batchRangesKernel(const float* __restrict__ a0, const float* __restrict__ a1,
                                  const float* __restrict__ a2, size_t n, size_t chunk,
                                  const uint64_t* __restrict__ first, uint32_t numSystems, uint32_t* __restrict__ out,
                                  unsigned stride)
{
    const float* const arrays[3] = {a0, a1, a2};
    const unsigned lane          = laneId();
    const size_t c0 = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) / kWarp * chunk;
    if (c0 >= n) return;
    const size_t c1 = c0 + chunk < n ? c0 + chunk : n;
    uint32_t sys    = systemOf(first, numSystems, c0);
    for (size_t pos = c0; pos < c1; ++sys)
    {
        const uint64_t end = __ldg(first + sys + 1);
        if (end <= pos) continue; // an empty system
        const size_t last = end < c1 ? size_t(end) : c1;
        uint32_t lo[kArrays], hi[kArrays];
#pragma unroll
        for (int k = 0; k < kArrays; ++k)
        {
            lo[k] = kSkipNaN ? orderedBits(INFINITY) : 0xffffffffu;
            hi[k] = kSkipNaN ? orderedBits(-INFINITY) : 0u;
        }
        for (; pos < last; pos += kRangeStep)
        {
#pragma unroll
            for (int j = 0; j < kRangeStep / kWarp; ++j)
            {
                const size_t i = pos + j * kWarp + lane;
                if (i >= last) continue;
#pragma unroll
                for (int k = 0; k < kArrays; ++k)
                {
                    const float v    = arrays[k][i];
                    const uint32_t u = orderedBits(v);
                    if (kSkipNaN && isnan(v)) continue;
                    lo[k] = min(lo[k], u);
                    hi[k] = max(hi[k], u);
                }
            }
        }
        pos = last;
#pragma unroll
        for (int k = 0; k < kArrays; ++k)
        {
            lo[k] = __reduce_min_sync(0xffffffffu, lo[k]);
            hi[k] = __reduce_max_sync(0xffffffffu, hi[k]);
            if (lane == 2 * k) atomicMin(out + size_t(sys) * stride + 2 * k, lo[k]);
            if (lane == 2 * k + 1) atomicMax(out + size_t(sys) * stride + 2 * k + 1, hi[k]);
        }
    }
}

template<int kArrays, bool kSkipNaN>
static void launchBatchRanges(const float* a0, const float* a1, const float* a2, size_t n, const uint64_t* first,
                              uint32_t numSystems, uint32_t* out, unsigned stride, cudaStream_t s)
{
    if (n == 0) return;
    // at most about 64 warps per SM, so that few atomics meet at a large system's values
    const size_t most   = size_t(kRangeStep) * 64 * 148;
    const size_t rounds = (n + most - 1) / most;
    const size_t chunk  = rounds * kRangeStep;
    const size_t warps  = (n + chunk - 1) / chunk;
    batchRangesKernel<kArrays, kSkipNaN><<<ceilDiv(warps * kWarp, 128), 128, 0, s>>>(a0, a1, a2, n, chunk, first,
                                                                                    numSystems, out, stride);
    RYO_LAUNCH_CHECK();
}

__global__ void batchMinMaxInit(uint32_t* mm, uint32_t numSystems)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 6 * numSystems) mm[i] = (i & 1) ? 0u : 0xffffffffu;
}

/*! the cube enclosing each system whose box is not given, as the single-system solve derives it: lower corner at the
 *  minimum, edge = largest extent (FP64), upper limit rounded up to cover the maximum */
__global__ void batchAutoBoxes(const uint32_t* __restrict__ mm, const int* __restrict__ useGiven, uint32_t numSystems,
                               DevBox<float>* __restrict__ boxes, float* __restrict__ limits)
{
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= numSystems || useGiven[s]) return;
    float mn[3], mx[3];
    double ext = 0.0;
    for (int d = 0; d < 3; ++d)
    {
        mn[d] = orderedFloat(mm[6 * s + 2 * d]);
        mx[d] = orderedFloat(mm[6 * s + 2 * d + 1]);
        ext   = fmax(ext, double(mx[d]) - double(mn[d]));
    }
    if (!(ext > 0)) ext = 1.0;
    DevBox<float> b;
    for (int d = 0; d < 3; ++d)
    {
        float lo = mn[d];
        float hi = float(double(mn[d]) + ext);
        if (!(hi >= mx[d])) hi = nextafterf(mx[d], 3.4e38f);
        limits[6 * s + 2 * d]     = lo;
        limits[6 * s + 2 * d + 1] = hi;
        b.lo[d]                   = lo;
        b.len[d]                  = hi - lo;
        b.inv[d]                  = 1.f / (hi - lo);
        b.bits[d]                 = kMaxLevel; // a cube: no axis is reduced
    }
    b.periodic = 0;
    boxes[s]   = b;
}

//! the two-level Hilbert tables (identical keys to hilbert3), built at compile time
static __device__ const HilbertLut kBatchHilbertLut = makeHilbertLut();

__global__ void __launch_bounds__(256) batchKeysKernel(const float* __restrict__ x, const float* __restrict__ y,
                                                       const float* __restrict__ z, size_t n,
                                                       const uint64_t* __restrict__ first, uint32_t numSystems,
                                                       const DevBox<float>* __restrict__ boxes, int sysBits,
                                                       uint64_t* __restrict__ keys)
{
    __shared__ uint16_t two[48 * 64];
    __shared__ uint16_t one[48 * 8];
    for (int i = threadIdx.x; i < 48 * 64; i += blockDim.x)
        two[i] = kBatchHilbertLut.two[i];
    for (int i = threadIdx.x; i < 48 * 8; i += blockDim.x)
        one[i] = kBatchHilbertLut.one[i];
    __syncthreads();
    size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
    {
        uint32_t s           = systemOf(first, numSystems, i);
        const DevBox<float>& b = boxes[s];
        unsigned ic[3];
        pointCells(x[i], y[i], z[i], b, ic);
        bool full  = b.bits[0] == unsigned(kMaxLevel) && b.bits[1] == unsigned(kMaxLevel) &&
                    b.bits[2] == unsigned(kMaxLevel);
        uint64_t k = full ? hilbert3Lut(ic[0], ic[1], ic[2], two, one) : hilbertKey(ic[0], ic[1], ic[2], b.bits);
        keys[i]    = (uint64_t(s) << (63 - sysBits)) | (k >> sysBits);
    }
}

/*! each system's root node (the level-L node of its prefix) and its first stack entry; flags a missing root */
__global__ void batchRootsKernel(uint32_t numSystems, const uint64_t* __restrict__ prefixes, int levelBegin,
                                 int levelEnd, const int* __restrict__ childOffsets, int sysLevel,
                                 const DevBox<float>* __restrict__ boxes, const int* __restrict__ numShells,
                                 SysTrav* __restrict__ out, int* __restrict__ rootNode, unsigned int* __restrict__ err)
{
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= numSystems) return;
    int sysBits     = 3 * sysLevel;
    uint64_t target = encodePrefix(uint64_t(s) << (63 - sysBits), sysBits);
    int lo = levelBegin, hi = levelEnd;
    while (lo < hi)
    {
        int mid = (lo + hi) >> 1;
        if (prefixes[mid] < target) lo = mid + 1;
        else hi = mid;
    }
    SysTrav t;
    if (lo < levelEnd && prefixes[lo] == target)
    {
        int fc  = childOffsets[lo];
        t.entry = fc != 0 ? fc : -(lo + 2);
        if (rootNode) rootNode[s] = lo;
    }
    else
    {
        t.entry = -1; // nothing to traverse; reported as an error
        if (rootNode) rootNode[s] = -1;
        atomicExch(err, 1u);
    }
    t.numShells = numShells[s];
    t.boxL[0]   = boxes[s].len[0];
    t.boxL[1]   = boxes[s].len[1];
    t.boxL[2]   = boxes[s].len[2];
    t.hLo       = 0xffffffffu; // filled by launchBatchSofteningRange
    t.hHi       = 0u;
    t.mLo       = 0xffffffffu;
    t.mHi       = 0u;
    out[s]      = t;
}

//! fixed groups of at most @p groupSize bodies inside every system
__global__ void batchGroupsKernel(uint32_t numGroups, const uint64_t* __restrict__ first,
                                  const uint32_t* __restrict__ groupOffset, uint32_t numSystems, uint32_t groupSize,
                                  uint32_t* __restrict__ start, uint32_t* __restrict__ end, uint32_t* __restrict__ sys)
{
    uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= numGroups) return;
    uint32_t lo = 0, hi = numSystems - 1;
    while (lo < hi)
    {
        uint32_t mid = (lo + hi + 1) >> 1;
        if (groupOffset[mid] <= g) lo = mid;
        else hi = mid - 1;
    }
    uint64_t b  = first[lo] + uint64_t(g - groupOffset[lo]) * groupSize;
    uint64_t e  = b + groupSize;
    uint64_t se = first[lo + 1];
    start[g]    = uint32_t(b);
    end[g]      = uint32_t(e < se ? e : se);
    sys[g]      = lo;
}

void launchBatchBoxes(const float* x, const float* y, const float* z, size_t n, const uint64_t* first,
                      uint32_t numSystems, const int* useGiven, uint32_t* mm, DevBox<float>* boxes, float* limits,
                      cudaStream_t s)
{
    batchMinMaxInit<<<ceilDiv(6 * numSystems, 256), 256, 0, s>>>(mm, numSystems);
    RYO_LAUNCH_CHECK();
    launchBatchRanges<3, true>(x, y, z, n, first, numSystems, mm, 6, s);
    batchAutoBoxes<<<ceilDiv(numSystems, 128), 128, 0, s>>>(mm, useGiven, numSystems, boxes, limits);
    RYO_LAUNCH_CHECK();
}

void launchBatchKeys(const float* x, const float* y, const float* z, size_t n, const uint64_t* first,
                     uint32_t numSystems, const DevBox<float>* boxes, int sysLevel, uint64_t* keys, int smCount,
                     cudaStream_t s)
{
    size_t want = ceilDiv(n, 256);
    size_t cap  = size_t(smCount) * 16;
    batchKeysKernel<<<unsigned(want < cap ? want : cap), 256, 0, s>>>(x, y, z, n, first, numSystems, boxes,
                                                                      3 * sysLevel, keys);
    RYO_LAUNCH_CHECK();
}

void launchBatchSofteningRange(const float* h, const float* m, size_t n, const uint64_t* first, uint32_t numSystems,
                               SysTrav* trav, cudaStream_t s)
{
    static_assert(offsetof(SysTrav, mHi) == offsetof(SysTrav, hLo) + 12 && sizeof(SysTrav) % 4 == 0);
    uint32_t* out         = reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(trav) + offsetof(SysTrav, hLo));
    const unsigned stride = sizeof(SysTrav) / 4;
    if (m) launchBatchRanges<2, false>(h, m, nullptr, n, first, numSystems, out, stride, s);
    else launchBatchRanges<1, false>(h, nullptr, nullptr, n, first, numSystems, out, stride, s);
}

void launchBatchRoots(uint32_t numSystems, const uint64_t* prefixes, int levelBegin, int levelEnd,
                      const int* childOffsets, int sysLevel, const DevBox<float>* boxes, const int* numShells,
                      SysTrav* out, int* rootNode, unsigned int* err, cudaStream_t s)
{
    batchRootsKernel<<<ceilDiv(numSystems, 128), 128, 0, s>>>(numSystems, prefixes, levelBegin, levelEnd, childOffsets,
                                                               sysLevel, boxes, numShells, out, rootNode, err);
    RYO_LAUNCH_CHECK();
}

void launchBatchGroups(uint32_t numGroups, const uint64_t* first, const uint32_t* groupOffset, uint32_t numSystems,
                       uint32_t groupSize, uint32_t* start, uint32_t* end, uint32_t* sys, cudaStream_t s)
{
    if (numGroups == 0) return;
    batchGroupsKernel<<<ceilDiv(numGroups, 256), 256, 0, s>>>(numGroups, first, groupOffset, numSystems, groupSize,
                                                              start, end, sys);
    RYO_LAUNCH_CHECK();
}

} // namespace ryo
