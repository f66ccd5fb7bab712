/*
 * ryoanji-b200: direct sums.
 *
 * ryo_direct_sum_* follow ryoanji/src/ryoanji/nbody/direct.cuh:36-107 (tiled all-pairs, P2P with the exact
 * 1/sqrt of the type, no G, p += m phi). The accuracy reference (launchDirectTargets) evaluates chosen targets of
 * float data entirely in double precision, the FP64 oracle that tree errors are quoted against; sources are staged
 * through shared memory in tiles and every thread owns one target.
 *
 * The float sum is bound by the FP32 pipe (13 packed operations per source and pair of targets): every lane owns two
 * targets in packed f32x2, as in the tree traversal, and the sources are split over the blocks of a cluster, which adds
 * its blocks' sums through distributed shared memory, so that a few thousand targets fill the GPU too. All pairs of
 * 40,001 bodies: 0.94 ms, against 2.60 ms with a target per thread and scalar arithmetic.
 */
#include <cfloat>
#include <cooperative_groups.h>

#include "internal.hpp"
#include "packed.cuh"

namespace ryo
{

constexpr int kDirectThreads = 256;

template<class T>
__device__ inline T exactRsqrt(T v);
template<>
__device__ inline double exactRsqrt<double>(double v)
{
    return rsqrt(v);
}

template<class T>
__device__ inline void p2pExact(T acc[4], const T ti[3], const T sj[3], T mj, T hi, T hj)
{
    T dx = sj[0] - ti[0], dy = sj[1] - ti[1], dz = sj[2] - ti[2];
    T R2    = dx * dx + (dy * dy + dz * dz);
    T hij   = hi + hj;
    T hij2  = hij * hij;
    T R2eff = (R2 < hij2) ? hij2 : R2;
    T invR  = exactRsqrt(R2eff);
    T m3    = mj * invR * (invR * invR);
    acc[0] -= m3 * R2;
    acc[1] += dx * m3;
    acc[2] += dy * m3;
    acc[3] += dz * m3;
}

template<class T>
__global__ void __launch_bounds__(kDirectThreads) directKernel(size_t first, size_t last, size_t numSource,
                                                               T sx, T sy, T sz, int numShells,
                                                               const T* __restrict__ x, const T* __restrict__ y,
                                                               const T* __restrict__ z, const T* __restrict__ m,
                                                               const T* __restrict__ h, T* p, T* ax, T* ay, T* az)
{
    __shared__ T tile[kDirectThreads][5];
    size_t t  = first + size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    T pos[3]  = {T(0), T(0), T(0)};
    T hi      = T(1);
    if (t < last)
    {
        pos[0] = x[t];
        pos[1] = y[t];
        pos[2] = z[t];
        hi     = h[t];
    }
    T acc[4] = {T(0), T(0), T(0), T(0)};
    for (int iz = -numShells; iz <= numShells; ++iz)
        for (int iy = -numShells; iy <= numShells; ++iy)
            for (int ix = -numShells; ix <= numShells; ++ix)
            {
                T ti[3] = {pos[0] + ix * sx, pos[1] + iy * sy, pos[2] + iz * sz};
                for (size_t s0 = 0; s0 < numSource; s0 += kDirectThreads)
                {
                    size_t j = s0 + threadIdx.x;
                    if (j < numSource)
                    {
                        tile[threadIdx.x][0] = x[j];
                        tile[threadIdx.x][1] = y[j];
                        tile[threadIdx.x][2] = z[j];
                        tile[threadIdx.x][3] = m[j];
                        tile[threadIdx.x][4] = h[j];
                    }
                    else
                    {
                        tile[threadIdx.x][0] = tile[threadIdx.x][1] = tile[threadIdx.x][2] = T(0);
                        tile[threadIdx.x][3] = T(0);
                        tile[threadIdx.x][4] = T(1);
                    }
                    __syncthreads();
                    for (int k = 0; k < kDirectThreads; ++k)
                    {
                        T sj[3] = {tile[k][0], tile[k][1], tile[k][2]};
                        p2pExact(acc, ti, sj, tile[k][3], hi, tile[k][4]);
                    }
                    __syncthreads();
                }
            }
    if (t < last)
    {
        if (p) p[t] += m[t] * acc[0];
        ax[t] += acc[1];
        ay[t] += acc[2];
        az[t] += acc[3];
    }
}

constexpr int kPackedThreads = 128;
constexpr int kPackedTargets = 2 * kPackedThreads; // per block
constexpr int kPackedTile    = 128;                // sources staged at a time, one per thread
constexpr int kPackedBlocks  = 9;                  // resident blocks per SM
constexpr int kMaxSplit      = 8;                  // blocks of a cluster, each with its share of the sources

//! max that keeps a NaN of @p r2, as the comparison r2 < hh ? hh : r2 does (hh is no NaN)
__device__ __forceinline__ float maxNan(float r2, float hh)
{
    float v;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(v) : "f"(r2), "f"(hh));
    return v;
}

struct PackedSum
{
    f2 p, x, y, z; // sum of m r^2 / r^3 (-phi), accelerations
};

//! both targets against one source; kNormal: the softening floor is a normal float, which the flushing rsqrt keeps
template<bool kNormal>
__device__ __forceinline__ void packedPair(PackedSum& A, f2 tx, f2 ty, f2 tz, float h0, float h1, f2 sx, f2 sy, f2 sz,
                                           f2 sm)
{
    f2 dx = sub2(sx, tx), dy = sub2(sy, ty), dz = sub2(sz, tz);
    f2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
    float a, b;
    upk(r2, a, b);
    a     = maxNan(a, h0);
    b     = maxNan(b, h1);
    f2 ir = kNormal ? pk(rsqrtApprox(a), rsqrtApprox(b)) : pk(rsqrtf(a), rsqrtf(b));
    f2 m3 = mul2(mul2(sm, ir), mul2(ir, ir));
    A.p   = fma2(m3, r2, A.p);
    A.x   = fma2(m3, dx, A.x);
    A.y   = fma2(m3, dy, A.y);
    A.z   = fma2(m3, dz, A.z);
}

//! (h_i + h_j)^2, or 0 for a NaN, which every comparison passes over
__device__ __forceinline__ float softeningFloor(float hi, float hj)
{
    const float s = hi + hj, q = s * s;
    return q == q ? q : 0.f;
}

__global__ void __launch_bounds__(kPackedThreads, kPackedBlocks)
    directPackedKernel(size_t first, size_t last, size_t numSource, float Lx, float Ly, float Lz, int numShells,
                       const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ z,
                       const float* __restrict__ m, const float* __restrict__ h, float* p, float* ax, float* ay,
                       float* az)
{
    __shared__ float4 tile[2 * kPackedTile]; // (x, x, y, y), (z, z, m, m)
    __shared__ float tileH[kPackedTile];
    __shared__ float4 sums[kPackedTargets];
    namespace cg         = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const unsigned split = cl.block_rank(), splits = cl.num_blocks();
    const size_t s0 = numSource * split / splits, s1 = numSource * (split + 1) / splits;
    const size_t base = first + size_t(blockIdx.x / splits) * kPackedTargets;
    // a thread's targets are base + tid and base + tid + kPackedThreads; those past the end repeat the last one
    const size_t i0 = min(base + threadIdx.x, last - 1), i1 = min(base + kPackedThreads + threadIdx.x, last - 1);
    const float h0 = h[i0], h1 = h[i1];
    PackedSum total{0ull, 0ull, 0ull, 0ull};
    for (int iz = -numShells; iz <= numShells; ++iz)
        for (int iy = -numShells; iy <= numShells; ++iy)
            for (int ix = -numShells; ix <= numShells; ++ix)
            {
                const f2 tx = pk(x[i0] + ix * Lx, x[i1] + ix * Lx), ty = pk(y[i0] + iy * Ly, y[i1] + iy * Ly),
                         tz = pk(z[i0] + iz * Lz, z[i1] + iz * Lz);
                for (size_t s = s0; s < s1; s += kPackedTile)
                {
                    const size_t j  = s + threadIdx.x;
                    const int count = int(min(size_t(kPackedTile), s1 - s));
                    const float hj  = j < s1 ? h[j] : h0;
                    if (j < s1)
                    {
                        const float sx = x[j], sy = y[j], sz = z[j], sm = m[j];
                        tile[2 * threadIdx.x]     = make_float4(sx, sx, sy, sy);
                        tile[2 * threadIdx.x + 1] = make_float4(sz, sz, sm, sm);
                        tileH[threadIdx.x]        = hj;
                    }
                    // the barrier that publishes the tile also asks whether one softening holds for it and its targets
                    const float hh  = softeningFloor(h0, h0);
                    const bool same = __syncthreads_and(hj == h0 && h1 == h0 && hh >= FLT_MIN) &&
                                      __syncthreads_and(h0 == tileH[0]);
                    PackedSum a{0ull, 0ull, 0ull, 0ull}, b = a;
                    auto source = [&](PackedSum& A, int k, bool uniform)
                    {
                        const ulonglong2 u = reinterpret_cast<const ulonglong2*>(tile)[2 * k];
                        const ulonglong2 v = reinterpret_cast<const ulonglong2*>(tile)[2 * k + 1];
                        if (uniform) packedPair<true>(A, tx, ty, tz, hh, hh, u.x, u.y, v.x, v.y);
                        else
                            packedPair<false>(A, tx, ty, tz, softeningFloor(h0, tileH[k]),
                                              softeningFloor(h1, tileH[k]), u.x, u.y, v.x, v.y);
                    };
                    if (same && count == kPackedTile)
                    {
#pragma unroll 4
                        for (int k = 0; k < kPackedTile; k += 2)
                        {
                            source(a, k, true);
                            source(b, k + 1, true);
                        }
                    }
                    else
                        for (int k = 0; k < count; ++k)
                            source(a, k, same);
                    total.p = add2(total.p, add2(a.p, b.p));
                    total.x = add2(total.x, add2(a.x, b.x));
                    total.y = add2(total.y, add2(a.y, b.y));
                    total.z = add2(total.z, add2(a.z, b.z));
                    __syncthreads();
                }
            }
    float q[4][2];
    upk(total.p, q[0][0], q[0][1]);
    upk(total.x, q[1][0], q[1][1]);
    upk(total.y, q[2][0], q[2][1]);
    upk(total.z, q[3][0], q[3][1]);
    sums[threadIdx.x]                  = make_float4(q[0][0], q[1][0], q[2][0], q[3][0]);
    sums[kPackedThreads + threadIdx.x] = make_float4(q[0][1], q[1][1], q[2][1], q[3][1]);
    cl.sync();
    // each block adds up its share of the cluster's targets
    const unsigned share = kPackedTargets / splits;
    for (unsigned k = split * share + threadIdx.x; k < (split + 1) * share; k += kPackedThreads)
    {
        double r[4] = {0.0, 0.0, 0.0, 0.0};
        for (unsigned c = 0; c < splits; ++c)
        {
            const float4 v = cl.map_shared_rank(sums, c)[k];
            r[0] += v.x;
            r[1] += v.y;
            r[2] += v.z;
            r[3] += v.w;
        }
        const size_t t = base + k;
        if (t < last)
        {
            if (p) p[t] += m[t] * float(-r[0]);
            ax[t] += float(r[1]);
            ay[t] += float(r[2]);
            az[t] += float(r[3]);
        }
    }
    cl.sync(); // a block's sums stay until every block has read them
}

static void launchDirectPacked(size_t first, size_t last, size_t numBodies, const float L[3], int numShells,
                               const float* x, const float* y, const float* z, const float* m, const float* h, float* p,
                               float* ax, float* ay, float* az, cudaStream_t s)
{
    // as many blocks per cluster as fill the GPU (eight per SM) with the targets there are, each with at least a tile
    // of sources; up to nine per SM are resident, so that a little more than eight still runs as one wave
    const unsigned blocks = ceilDiv(last - first, kPackedTargets);
    unsigned splits       = 1;
    while (splits < unsigned(kMaxSplit) && blocks * splits < 8 * 148 && numBodies / (2 * splits) >= kPackedTile)
        splits *= 2;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim  = dim3(blocks * splits);
    cfg.blockDim = dim3(kPackedThreads);
    cfg.stream   = s;
    cudaLaunchAttribute attr{};
    attr.id               = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = splits;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs    = &attr;
    cfg.numAttrs = 1;
    RYO_CUDA(cudaLaunchKernelEx(&cfg, directPackedKernel, first, last, numBodies, L[0], L[1], L[2], numShells, x, y, z,
                                m, h, p, ax, ay, az));
    RYO_LAUNCH_CHECK();
}

template<class T>
void launchDirect(size_t first, size_t last, size_t numBodies, const T* boxL, int numShells, const T* x, const T* y,
                  const T* z, const T* m, const T* h, T* p, T* ax, T* ay, T* az, cudaStream_t s)
{
    if (last <= first) return;
    T L[3] = {boxL ? boxL[0] : T(0), boxL ? boxL[1] : T(0), boxL ? boxL[2] : T(0)};
    if constexpr (sizeof(T) == 4)
        launchDirectPacked(first, last, numBodies, L, numShells, x, y, z, m, h, p, ax, ay, az, s);
    else
    {
        directKernel<T><<<ceilDiv(last - first, kDirectThreads), kDirectThreads, 0, s>>>(
            first, last, numBodies, L[0], L[1], L[2], numShells, x, y, z, m, h, p, ax, ay, az);
        RYO_LAUNCH_CHECK();
    }
}

template void launchDirect<float>(size_t, size_t, size_t, const float*, int, const float*, const float*,
                                  const float*, const float*, const float*, float*, float*, float*, float*,
                                  cudaStream_t);
template void launchDirect<double>(size_t, size_t, size_t, const double*, int, const double*, const double*,
                                   const double*, const double*, const double*, double*, double*, double*, double*,
                                   cudaStream_t);

//! double-precision reference for chosen targets; sources in float are staged as float4 + h
__global__ void __launch_bounds__(kDirectThreads) directTargetsKernel(const int64_t* __restrict__ targets,
                                                                      size_t numTargets, const float* __restrict__ x,
                                                                      const float* __restrict__ y,
                                                                      const float* __restrict__ z,
                                                                      const float* __restrict__ m,
                                                                      const float* __restrict__ h, size_t numBodies,
                                                                      double G, double Lx, double Ly, double Lz,
                                                                      int numShells, double* pot, double* ax,
                                                                      double* ay, double* az)
{
    __shared__ float4 tile[kDirectThreads];
    __shared__ float tileH[kDirectThreads];
    size_t t  = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    int64_t i = t < numTargets ? targets[t] : 0;
    double pos[3] = {double(x[i]), double(y[i]), double(z[i])};
    double hi     = h[i];
    double acc[4] = {0, 0, 0, 0};
    for (int iz = -numShells; iz <= numShells; ++iz)
        for (int iy = -numShells; iy <= numShells; ++iy)
            for (int ix = -numShells; ix <= numShells; ++ix)
            {
                double ti[3] = {pos[0] + ix * Lx, pos[1] + iy * Ly, pos[2] + iz * Lz};
                for (size_t s0 = 0; s0 < numBodies; s0 += kDirectThreads)
                {
                    size_t j = s0 + threadIdx.x;
                    if (j < numBodies)
                    {
                        tile[threadIdx.x]  = make_float4(x[j], y[j], z[j], m[j]);
                        tileH[threadIdx.x] = h[j];
                    }
                    else
                    {
                        tile[threadIdx.x]  = make_float4(0.f, 0.f, 0.f, 0.f);
                        tileH[threadIdx.x] = 1.f;
                    }
                    __syncthreads();
                    int cnt = int(numBodies - s0 < size_t(kDirectThreads) ? numBodies - s0 : kDirectThreads);
                    for (int k = 0; k < cnt; ++k)
                    {
                        float4 sj4   = tile[k];
                        double sj[3] = {sj4.x, sj4.y, sj4.z};
                        p2pExact<double>(acc, ti, sj, double(sj4.w), hi, double(tileH[k]));
                    }
                    __syncthreads();
                }
            }
    if (t < numTargets)
    {
        pot[t] = G * double(m[i]) * acc[0];
        ax[t]  = G * acc[1];
        ay[t]  = G * acc[2];
        az[t]  = G * acc[3];
    }
}

void launchDirectTargets(const int64_t* targets, size_t numTargets, const float* x, const float* y, const float* z,
                         const float* m, const float* h, size_t numBodies, double G, const double* boxL,
                         int numShells, double* pot, double* ax, double* ay, double* az, cudaStream_t s)
{
    if (numTargets == 0) return;
    double L[3] = {boxL ? boxL[0] : 0.0, boxL ? boxL[1] : 0.0, boxL ? boxL[2] : 0.0};
    directTargetsKernel<<<ceilDiv(numTargets, kDirectThreads), kDirectThreads, 0, s>>>(
        targets, numTargets, x, y, z, m, h, numBodies, G, L[0], L[1], L[2], numShells, pot, ax, ay, az);
    RYO_LAUNCH_CHECK();
}

} // namespace ryo
