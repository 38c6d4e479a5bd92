// mgr_common.cuh — device helpers shared by the 2D and 3D kernels of
// libmgr (B-spline registration cost+gradient on sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace mgr {

// ---------------------------------------------------------------------
// cubic B-spline arithmetic
// ---------------------------------------------------------------------

// Start index of the 4-tap window of a coordinate, with the reference's
// fixed-point floor: the coordinate is rounded to the nearest multiple of
// 2^-16 (ties to even) before flooring (mia/core/splinekernel.cc:164-192,
// 250-255).  For a float coordinate, x*65536 is exact and rint() rounds it
// exactly as the reference's 1.5*2^36 double trick does.
__device__ __forceinline__ int ffloor16(float x)
{
    return __float2int_rn(x * 65536.0f) >> 16;
}

// Cubic B-spline weights at fractional offset f, in the reference's
// evaluation order (mia/core/splinekernel/bspline.cc:258-285).
__device__ __forceinline__ void bspline3_weights(float f, float w[4])
{
    const float ob6 = 1.0f / 6.0f;
    const float xm1 = 1.0f - f;
    const float w0 = (xm1 * xm1) * (xm1 * ob6);
    const float w3 = (f * f) * (f * ob6);
    w[0] = w0;
    w[3] = w3;
    w[1] = ((xm1 - w0) - w0) + w3;
    w[2] = ((f - w3) - w3) + w0;
}

// Mirror halo of the padded copy of the prefiltered moving image that the
// split path's warp kernel stages from (voxels per side; the padded rows are
// 128-byte aligned so that any 16-byte aligned row segment can be copied
// with one bulk copy).
constexpr int PAD_H = 16;

__host__ __device__ inline int pad_pitch(int nx)
{
    return ((nx + 2 * PAD_H + 31) / 32) * 32;
}

// Mirror boundary index folding with period 2w-2
// (mia/core/splinebc/bc.cc:52-64).
__device__ __forceinline__ int mirror_fold(int i, int w)
{
    const int w2 = 2 * w - 2;
    int idx = i < 0 ? -i : i;
    idx = (w == 1) ? 0 : ((idx < w2) ? idx : idx % w2);
    if (w <= idx) idx = w2 - idx;
    return idx;
}

// clamp to [mn, mx] with the reference's comparison order
// (bounded<>, mia/3d/interpolator.cxx:177-185)
__device__ __forceinline__ float clamp_ref(float r, float mn, float mx)
{
    return (r >= mn) ? ((r <= mx) ? r : mx) : mn;
}

// Tricubic B-spline interpolation of a prefiltered volume at p, mirror BC.
__device__ __forceinline__ float sample3(const float *__restrict__ c, int nx, int ny, int nz,
                                         float px, float py, float pz, float mn, float mx)
{
    const int fx = ffloor16(px), fy = ffloor16(py), fz = ffloor16(pz);
    float wx[4], wy[4], wz[4];
    bspline3_weights(px - float(fx), wx);
    bspline3_weights(py - float(fy), wy);
    bspline3_weights(pz - float(fz), wz);
    int ix[4], iy[4], iz[4];
    const int sx = fx - 1, sy = fy - 1, sz = fz - 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        ix[k] = sx + k;
        iy[k] = sy + k;
        iz[k] = sz + k;
    }
    // the mirror fold runs only near the border (a real branch, so the
    // interior path does not pay for the modulo)
    if (sx < 0 || sx + 3 >= nx) {
#pragma unroll
        for (int k = 0; k < 4; ++k) ix[k] = mirror_fold(ix[k], nx);
    }
    if (sy < 0 || sy + 3 >= ny) {
#pragma unroll
        for (int k = 0; k < 4; ++k) iy[k] = mirror_fold(iy[k], ny);
    }
    if (sz < 0 || sz + 3 >= nz) {
#pragma unroll
        for (int k = 0; k < 4; ++k) iz[k] = mirror_fold(iz[k], nz);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) iy[k] *= nx;
    const size_t nxy = size_t(nx) * ny;
    float acc = 0.0f;
#pragma unroll
    for (int kz = 0; kz < 4; ++kz) {
        const float *__restrict__ pl = c + size_t(iz[kz]) * nxy;
        float ay = 0.0f;
#pragma unroll
        for (int ky = 0; ky < 4; ++ky) {
            const float *__restrict__ row = pl + iy[ky];
            const float r = wx[0] * __ldg(row + ix[0]) + wx[1] * __ldg(row + ix[1]) +
                            wx[2] * __ldg(row + ix[2]) + wx[3] * __ldg(row + ix[3]);
            ay += wy[ky] * r;
        }
        acc += wz[kz] * ay;
    }
    return clamp_ref(acc, mn, mx);
}

// Bicubic variant (mia/2d/interpolator.cxx:216-311).
__device__ __forceinline__ float sample2(const float *__restrict__ c, int nx, int ny, float px,
                                         float py, float mn, float mx)
{
    const int fx = ffloor16(px), fy = ffloor16(py);
    float wx[4], wy[4];
    bspline3_weights(px - float(fx), wx);
    bspline3_weights(py - float(fy), wy);
    int ix[4], iy[4];
    const int sx = fx - 1, sy = fy - 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        ix[k] = sx + k;
        iy[k] = sy + k;
    }
    if (sx < 0 || sx + 3 >= nx) {
#pragma unroll
        for (int k = 0; k < 4; ++k) ix[k] = mirror_fold(ix[k], nx);
    }
    if (sy < 0 || sy + 3 >= ny) {
#pragma unroll
        for (int k = 0; k < 4; ++k) iy[k] = mirror_fold(iy[k], ny);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) iy[k] *= nx;
    float acc = 0.0f;
#pragma unroll
    for (int ky = 0; ky < 4; ++ky) {
        const float *__restrict__ row = c + iy[ky];
        const float r = wx[0] * __ldg(row + ix[0]) + wx[1] * __ldg(row + ix[1]) +
                        wx[2] * __ldg(row + ix[2]) + wx[3] * __ldg(row + ix[3]);
        acc += wy[ky] * r;
    }
    return clamp_ref(acc, mn, mx);
}

// Bicubic sample whose first tap (fx-1, fy-1) is at `base`, rows `sy` floats
// apart, no index folding needed.  Same weights and summation order as
// sample2.
__device__ __forceinline__ float sample2_at(const float *base, int sy, float px, float py, int fx, int fy,
                                                float mn, float mx)
{
    float wx[4], wy[4];
    bspline3_weights(px - float(fx), wx);
    bspline3_weights(py - float(fy), wy);
    float acc = 0.0f;
#pragma unroll
    for (int ky = 0; ky < 4; ++ky) {
        const float *row = base + ky * sy;
        const float r = wx[0] * row[0] + wx[1] * row[1] + wx[2] * row[2] + wx[3] * row[3];
        acc += wy[ky] * r;
    }
    return clamp_ref(acc, mn, mx);
}

// ---------------------------------------------------------------------
// Pairs of floats in a 64-bit register pair: one instruction does the
// arithmetic of both, each rounded as its scalar form rounds.
// ---------------------------------------------------------------------
typedef unsigned long long float2x;

__device__ __forceinline__ float2x pack2(float a, float b)
{
    float2x r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(float2x v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ float2x add2(float2x a, float2x b)
{
    float2x r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float2x add2_down(float2x a, float2x b)
{
    float2x r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float2x sub2(float2x a, float2x b)
{
    float2x r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float2x mul2(float2x a, float2x b)
{
    float2x r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float2x fma2(float2x a, float2x b, float2x c)
{
    float2x r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// ---------------------------------------------------------------------
// programmatic dependent launch
// ---------------------------------------------------------------------
// A kernel launched with cudaLaunchAttributeProgrammaticStreamSerialization
// may start while the kernel before it in the stream is still running;
// pdl_wait returns once that kernel has completed and its writes are visible
// (at once for a kernel launched without the attribute).  Before it a kernel
// reads only the level's fixed tables.  pdl_trigger, issued by every block
// after its pdl_wait, lets the next kernel be launched: so no kernel starts
// before the one two places back in the stream has completed.  A kernel that
// triggers without a wait (the parameters' conversion) must be launched
// without the attribute, in plain stream order.
__device__ __forceinline__ void pdl_wait()
{
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}
__device__ __forceinline__ void pdl_trigger()
{
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// ---------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------
// double(x) with integer instructions: conversions to double share the FP64
// pipe, which runs at a small fraction of the FP32 rate
__device__ __forceinline__ double widen(float x)
{
    const unsigned u = __float_as_uint(x), m = u & 0x7fffffffu;
    if (m - 0x00800000u < 0x7f000000u)   // a normal number: the exponent's bias moves by 1023 - 127
        return __hiloint2double(int((u & 0x80000000u) | ((m >> 3) + 0x38000000u)), int(u << 29));
    return m == 0u ? __hiloint2double(int(u), 0) : double(x);
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums over the warp, each with warp_sum's tree (the same bits).  FP64
// additions issue at 1/64 of the FP32 rate here and several sums by every
// lane are what a reduction's time goes to, so lanes exchange halves of the
// values: a step adds each pair once instead of in both lanes.
//
// Two sums, 5 additions per lane instead of 10: sum 0 in lanes 0-15, sum 1 in
// lanes 16-31.
__device__ __forceinline__ double warp_sum2(double x0, double x1, int lane)
{
    const bool h16 = lane & 16;
    double a = (h16 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, h16 ? x0 : x1, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// Five sums, 11 additions instead of 25: even lanes hold sum (lane >> 3) & 3
// of the first four, odd lanes sum 4.
__device__ __forceinline__ double warp_sum5(const double (&x)[5], int lane)
{
    const bool h16 = lane & 16, h8 = lane & 8;
    double a = (h16 ? x[2] : x[0]) + __shfl_xor_sync(0xffffffffu, h16 ? x[0] : x[2], 16);
    const double b = (h16 ? x[3] : x[1]) + __shfl_xor_sync(0xffffffffu, h16 ? x[1] : x[3], 16);
    a = (h8 ? b : a) + __shfl_xor_sync(0xffffffffu, h8 ? a : b, 8);
    a += __shfl_xor_sync(0xffffffffu, a, 4);
    a += __shfl_xor_sync(0xffffffffu, a, 2);
    a += __shfl_xor_sync(0xffffffffu, a, 1);
    const double e = warp_sum(x[4]);
    return lane & 1 ? e : a;
}

// Block-wide sums of K (1, 2 or 5) doubles per thread in a block of NW warps:
// a warp_sum tree per warp, then the same tree over the warps' sums.  Every
// lane of warp 0 holds the results after it; `scratch` holds K * NW doubles.
// Order is fixed, so the result is reproducible from run to run.
template <int K, int NW = 8>
__device__ __forceinline__ void block_sum(double (&v)[K], double *scratch)
{
    static_assert(K == 1 || K == 2 || K == 5, "the sums that are taken together");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if constexpr (K == 1) {
        const double s = warp_sum(v[0]);
        if (lane == 0) scratch[wid] = s;
    } else if constexpr (K == 2) {
        const double s = warp_sum2(v[0], v[1], lane);
        if ((lane & 15) == 0) scratch[(lane >> 4) * NW + wid] = s;
    } else {
        const double s = warp_sum5(v, lane);
        if ((lane & 7) == 0) scratch[(lane >> 3) * NW + wid] = s;
        if (lane == 1) scratch[4 * NW + wid] = s;
    }
    __syncthreads();
    if (NW != 8 && wid == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = warp_sum(lane < NW ? scratch[k * NW + lane] : 0.0);
    } else if (wid == 0) {
        // lane 8 k + w: sum k of warp w (k < 4), the last of five apart; the
        // tree's first steps would add zeros
#pragma unroll
        for (int h = 0; h < (K == 5 ? 2 : 1); ++h) {
            const int at = h * 4 * NW + lane;
            double s = at < K * NW ? scratch[at] : 0.0;
#pragma unroll
            for (int o = NW / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
#pragma unroll
            for (int k = h * 4; k < (K < h * 4 + 4 ? K : h * 4 + 4); ++k)
                v[k] = __shfl_sync(0xffffffffu, s, (k - h * 4) * NW);
        }
    }
    __syncthreads();
}

// K sums at a time: components 0 .. K - 1 of the elements t, t + step, ...
// below n of p (element i at p + i * stride) added to v in this order, in
// batches of B elements whose loads are all in flight together (values that
// other blocks wrote: read through the L2)
template <int B, int K>
__device__ __forceinline__ void strided_sums(const double *p, int n, int t, int step, int stride, double (&v)[K])
{
    for (; t < n; t += B * step) {
        double x[B][K];
#pragma unroll
        for (int j = 0; j < B; ++j)
#pragma unroll
            for (int k = 0; k < K; ++k)
                x[j][k] = t + j * step < n ? __ldcg(p + size_t(t + j * step) * stride + k) : 0.0;
#pragma unroll
        for (int j = 0; j < B; ++j)
            if (t + j * step < n)
#pragma unroll
                for (int k = 0; k < K; ++k) v[k] += x[j][k];
    }
}

// Arrival at a counter: true for the last of n.  What the thread wrote before
// it, and what its block wrote before the barrier before it, is visible to
// the last one and, after its next barrier, to its block.
__device__ __forceinline__ bool arrive_last(unsigned *counter, int n)
{
    unsigned before;
    asm volatile("atom.acq_rel.gpu.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(counter) : "memory");
    return before == unsigned(n - 1);
}

// ---------------------------------------------------------------------
// per-axis tables (built on the host, see tables.cc)
// ---------------------------------------------------------------------
struct Axis {
    const int *fs;      // forward start index per voxel coordinate
    const float4 *fw;   // forward weights (4th zero on the last voxel)
    const int *as;      // adjoint start per voxel coordinate
    const float4 *aw;   // adjoint weights (float rows of translate)
    const int2 *rows;   // per coefficient: voxel range [first, first+len)
    const int *ftile0;  // per tile: first coefficient of the forward footprint
    const int *atile0;  // per tile: first coefficient of the adjoint footprint
    const int2 *gtile;  // per coefficient: tiles [lo, hi] whose adjoint footprint holds it
    const int *glist;   // per coefficient: GATHER_LMAX offsets into the partial slots, this axis' part
    const int *glen;    // per coefficient: entries of glist (-1: longer than GATHER_LMAX)
    const int2 *win;    // per coefficient: voxels [lo, hi) whose four adjoint coefficients include it
    int n;              // voxels
    int nc;             // coefficients
    int t;              // tile length (voxels)
    int nt;             // number of tiles
    int fc;             // forward footprint length (max over tiles)
    int ac;             // adjoint footprint length (max over tiles)
};

// longest per-axis list of tiles whose adjoint footprint holds a coefficient
// that the gather reads from the tables (longer lists take a slower path)
constexpr int GATHER_LMAX = 24;
// planes of the 3D warp kernel's shared-memory tap ring (split3.cu); the
// tile-fit rule (mgr_level::tile_fits) counts them.  12 keeps three warp
// blocks per SM at the usual spacings (14 measured slower: 2 blocks per SM
// at rate 5)
#ifndef MGR_RING_PLANES
#define MGR_RING_PLANES 12
#endif
constexpr int WARP_RING_PLANES = MGR_RING_PLANES;

// scalars written by the cost finalisation (double[16])
enum {
    SC_VALUE = 0,      // image cost value() (unweighted), NCC with the 1e-10 threshold
    SC_FORCE_COST = 1, // force-pass cost (2D full cost returns this)
    // the force constants, SC_K1 .. SC_FSCALE, are read as one range
    SC_K1 = 2,         // NCC: 2*cov/(var_a*var_b)  (gradient helper, 1e-5 threshold)
    SC_K2 = 3,         // NCC: cov/var_a
    SC_MA = 4,         // NCC: mean of the warped image
    SC_MB = 5,         // NCC: mean of the reference
    SC_FSCALE = 6,     // SSD: force scale (1/N with norm, else 1)
    SC_PEN = 7,        // penalty value (unweighted)
    SC_COST_IMG = 8,   // weighted image cost
    SC_COST_PEN = 9,   // weighted penalty cost
    SC_NSLOTS = 16
};

}  // namespace mgr
