// prefilter.cu — cubic B-spline prefilter (causal/anticausal IIR, pole
// sqrt(3)-2, mirror boundary) and the image min/max used by the
// interpolator's clamp.  Restates T3DConvoluteInterpolator::prefilter
// (mia/3d/interpolator.cxx:98-164) with CSplineBoundaryCondition::filter_line
// (mia/core/boundary_conditions.cc:62-103) and CMirrorOnBoundary
// (mia/core/splinebc/bc.cc:67-88): x lines, then y lines, then z lines, each
// line filtered with the reference's operations (in float, see
// prefilter_line) and stored back as float.
#include <cudaTypedefs.h>

#include <algorithm>
#include "mgr_common.cuh"
#include "mgr_kernels.hh"

namespace mgr {

// One pass filters the lines of one axis; a block of PF_NT threads owns lb
// (<= 32) of them, staged in shared memory.  The loads come scaled by lambda
// (the filter's first step) and cover whole rows: along the line for x lines
// (a warp per line), across the lines (consecutive x) for y and z lines.  One
// thread per line then runs the recursion in two sweeps with the running
// value in a register, and the block stores the lines back.
//
// The passes also take what used to be passes of their own over the images:
// the first (x) reads the caller's image (no copy of it is made) and finds
// its minimum and maximum, the last writes the mirror-padded copy beside the
// coefficients.  What bounds a pass is the latency of load, recursion and
// store, one after the other in a block, so all its blocks are resident at
// once (eight of 32 lines on an SM), many loads are in flight and the
// recursion's loads run ahead of its chain: at 192x192x128 the recursion of a
// z line took 15.3 k cycles, 8.5 k now.  New images on a kept level and the
// evaluation after them, 192x192x128 SSD: 325 us with a kernel each for copy,
// bounds, means, three passes and padding, 180 us in three passes, 165 us so
// (169 with five blocks an SM, 172 with six, 167 with blocks of 128 threads).
//
// The reference filters each line in a double buffer; FP64 arithmetic runs
// at a small fraction of the FP32 rate on this GPU, so the recursion runs in
// float with the same operations: the pole's magnitude (0.268) damps the
// rounding of every step, and the result differs from the double filter by a
// few float ulp of the coefficient (the parity tests bound the warped image
// and costs, which read these coefficients, at 1e-5 / 1e-4).
constexpr int PF_NT = 256;
constexpr int PF_NW = PF_NT / 32;
constexpr int PF_BATCH = 8;   // line values a thread holds in registers at a time
constexpr int PF_MINB = 8;    // resident blocks per SM

struct PrefilterPass {
    const float *in;
    float *out;
    int n;               // line length
    int nlines;          // x pass: all lines; y and z passes: the image's x size
    int lb;              // lines per block, a power of two <= 32
    size_t estride;      // elements between neighbours of a line
    size_t bstride;      // y and z passes: elements between blockIdx.y groups
    // x pass: minimum and maximum of the input
    float2 *mmpart;      // one per block
    unsigned *counter;
    float *minmax;
    // last pass: the mirror-padded copy (null: none)
    float *pad;
    size_t pad_estride;  // its elements between neighbours of a line
    int pad_pitch;
    int ny;              // 3D: rows of a plane, blockIdx.y is the row; 2D: 0
};

// the line at c (elements s apart), already scaled by lambda
__device__ __forceinline__ void prefilter_line(float *c, int n, int s)
{
    const float p = float(1.7320508075688772 - 2.0);   // sqrt(3) - 2
    // mirror initial value: sum of (p^k + p^(2n-2-k)) c[k], k ascending; the
    // terms whose powers are below the float range add nothing, and from the
    // first of them on all following ones (short lines have no such term)
    float zn = p;
    const float iz = 1.0f / p;
    float z2n = powf(p, float(n - 1));
    float sum = c[0] + z2n * c[(n - 1) * s];
    z2n *= z2n * iz;
    // Each of the three walks goes in batches of PF_BATCH values, the next
    // batch's loads under way while this one's chain of dependent operations
    // runs: f(x) for each of the `count` values q[0], q[step], ...; store: the
    // value it returns in their place
    auto walk = [&](float *q, int step, int count, bool store, auto f, auto done) {
        if (count >= PF_BATCH) {
            float v[PF_BATCH];
#pragma unroll
            for (int j = 0; j < PF_BATCH; ++j) v[j] = q[j * step];
#pragma unroll 2
            for (; count >= 2 * PF_BATCH; count -= PF_BATCH) {
                float w[PF_BATCH];
                float *qn = q + PF_BATCH * step;
#pragma unroll
                for (int j = 0; j < PF_BATCH; ++j) w[j] = qn[j * step];
#pragma unroll
                for (int j = 0; j < PF_BATCH; ++j) v[j] = f(v[j]);
                if (done()) return;
#pragma unroll
                for (int j = 0; j < PF_BATCH; ++j) {
                    if (store) q[j * step] = v[j];
                    v[j] = w[j];
                }
                q = qn;
            }
#pragma unroll
            for (int j = 0; j < PF_BATCH; ++j) {
                const float r = f(v[j]);
                if (store) q[j * step] = r;
            }
            count -= PF_BATCH;
            q += PF_BATCH * step;
        }
        float v[PF_BATCH];
#pragma unroll
        for (int j = 0; j < PF_BATCH - 1; ++j) v[j] = j < count ? q[j * step] : 0.0f;
#pragma unroll
        for (int j = 0; j < PF_BATCH - 1; ++j)
            if (j < count) {
                const float r = f(v[j]);
                if (store) q[j * step] = r;
            }
    };
    auto never = [] { return false; };
    walk(c + s, s, n - 2, false,
         [&](float x) {
             sum += (zn + z2n) * x;
             zn *= p;
             z2n *= iz;
             return x;
         },
         [&] { return zn == 0.0f && z2n == 0.0f; });
    float prev = sum / (1.0f - zn * zn);
    c[0] = prev;
    walk(c + s, s, n - 1, true, [&](float x) { return prev = x + p * prev; }, never);
    const float before = c[max(n - 2, 0) * s];
    float next = (p / (p * p - 1.0f)) * (p * before + prev);
    c[(n - 1) * s] = next;
    walk(c + (n - 2) * s, -s, n - 1, true, [&](float x) { return next = p * (next - x); }, never);
}

__device__ __forceinline__ float prefilter_scale(float v)
{
    return v * float(2.0 - (1.7320508075688772 - 2.0) - 1.0 / (1.7320508075688772 - 2.0));
}

// x lines.  The minimum and maximum follow the reference's rule that the
// lower clamp bound is at most 0 (interpolator.cxx:109-112); the last block
// to finish reduces the blocks' values.
__global__ void __launch_bounds__(PF_NT, PF_MINB) k_prefilter_x(PrefilterPass a)
{
    extern __shared__ float sl[];
    __shared__ float2 wmm[PF_NW];
    __shared__ bool last;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int n = a.n, pitch = n | 1;
    const int l0 = blockIdx.x * a.lb, nl = min(a.lb, a.nlines - l0);
    const float *src = a.in + size_t(l0) * n;
    float mn = INFINITY, mx = -INFINITY;
    // (two lines of a warp at a time: more loads in flight)
    for (int l = w; l < nl; l += 2 * PF_NW) {
        const float *row = src + size_t(l) * n;
        float *c = sl + l * pitch;
        const bool two = l + PF_NW < nl;
        for (int k0 = lane; k0 < n; k0 += 32 * PF_BATCH) {
            float v[2][PF_BATCH];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < PF_BATCH; ++j)
                    v[i][j] = k0 + 32 * j < n && (i == 0 || two) ? __ldg(row + size_t(i) * PF_NW * n + k0 + 32 * j) : 0.0f;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < PF_BATCH; ++j)
                    if (k0 + 32 * j < n && (i == 0 || two)) {
                        mn = fminf(mn, v[i][j]);
                        mx = fmaxf(mx, v[i][j]);
                        c[i * PF_NW * pitch + k0 + 32 * j] = prefilter_scale(v[i][j]);
                    }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) wmm[w] = make_float2(mn, mx);
    __syncthreads();
    if (t < nl) prefilter_line(sl + t * pitch, n, 1);
    if (t == PF_NT - 1) {   // a thread without a line (lb <= 32)
        for (int k = 0; k < PF_NW; ++k) {
            mn = fminf(mn, wmm[k].x);
            mx = fmaxf(mx, wmm[k].y);
        }
        a.mmpart[blockIdx.x] = make_float2(mn, mx);
        __threadfence();
        last = atomicAdd(a.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    float *dst = a.out + size_t(l0) * n;
    for (int l = w; l < nl; l += PF_NW) {
        float *row = dst + size_t(l) * n;
        const float *c = sl + l * pitch;
#pragma unroll 4
        for (int k = lane; k < n; k += 32) row[k] = c[k];
    }
    if (!last) return;
    __threadfence();
    mn = INFINITY;
    mx = -INFINITY;
    for (unsigned i = t; i < gridDim.x; i += PF_NT) {
        const float2 v = __ldcg(a.mmpart + i);
        mn = fminf(mn, v.x);
        mx = fmaxf(mx, v.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) wmm[w] = make_float2(mn, mx);
    __syncthreads();
    if (t == 0) {
        for (int k = 0; k < PF_NW; ++k) {
            mn = fminf(mn, wmm[k].x);
            mx = fmaxf(mx, wmm[k].y);
        }
        if (0.0f < mn) mn = 0.0f;
        if (mx < mn) mx = mn;   // an image of NaN alone: its samples are the lower bound
        a.minmax[0] = mn;
        a.minmax[1] = mx;
        *a.counter = 0;
    }
}

// y or z lines of lb consecutive x, in place; PAD: the mirror-padded copy is
// written from the staged lines, every image of a line's elements along the
// line, of the row across the plane's rows (3D) and of the columns within
// PAD_H of the image's x borders
template <bool PAD>
__global__ void __launch_bounds__(PF_NT, PF_MINB) k_prefilter_cols(PrefilterPass a)
{
    extern __shared__ float sl[];
    __shared__ int images[2 * PAD_H + 1];   // PAD, 3D: the padded rows that hold this row
    __shared__ int nimages;
    const int t = threadIdx.x, n = a.n, lb = a.lb;
    const int xb = blockIdx.x * lb, nl = min(lb, a.nlines - xb);
    const int l = t & (lb - 1), g = t / lb, ng = PF_NT / lb;
    const size_t base = size_t(blockIdx.y) * a.bstride + xb + l;
    if (l < nl)
        for (int k0 = g; k0 < n; k0 += ng * 2 * PF_BATCH) {
            float v[2 * PF_BATCH];
#pragma unroll
            for (int j = 0; j < 2 * PF_BATCH; ++j)
                v[j] = k0 + ng * j < n ? __ldcg(a.in + base + size_t(k0 + ng * j) * a.estride) : 0.0f;
#pragma unroll
            for (int j = 0; j < 2 * PF_BATCH; ++j)
                if (k0 + ng * j < n) sl[(k0 + ng * j) * lb + l] = prefilter_scale(v[j]);
        }
    if (PAD && t >= PF_NT - 32) {   // the last warp has no line
        const int j = t & 31, yp = j < PAD_H ? j - PAD_H : a.ny + j - PAD_H;
        const bool hit = a.ny > 0 && mirror_fold(yp, a.ny) == int(blockIdx.y);
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) images[1 + __popc(m & ((1u << j) - 1u))] = yp + PAD_H;
        if (j == 0) {
            images[0] = a.ny > 0 ? int(blockIdx.y) + PAD_H : 0;
            nimages = 1 + __popc(m);
        }
    }
    __syncthreads();
    if (t < nl) prefilter_line(sl + t, n, lb);
    __syncthreads();
    if (!PAD) {
        if (l < nl) {
#pragma unroll 4
            for (int k = g; k < n; k += ng) a.out[base + size_t(k) * a.estride] = sl[k * lb + l];
        }
        return;
    }
    const int nimg = nimages, np = n + 2 * PAD_H, nx = a.nlines;
    if (l < nl) {
        // the coefficients, and each in the padded row of its own (most rows
        // have no other image)
        float *const col = a.pad + PAD_H + xb + l;
        float *const own = col + size_t(PAD_H) * a.pad_estride + size_t(images[0]) * a.pad_pitch;
#pragma unroll 4
        for (int k = g; k < n; k += ng) {
            const float v = sl[k * lb + l];
            a.out[base + size_t(k) * a.estride] = v;
            own[size_t(k) * a.pad_estride] = v;
        }
        // the other rows that hold this one
        if (nimg > 1)
            for (int k = g; k < n; k += ng) {
                const float v = sl[k * lb + l];
                for (int r = 1; r < nimg; ++r)
                    col[size_t(k + PAD_H) * a.pad_estride + size_t(images[r]) * a.pad_pitch] = v;
            }
        // the halo along the line
        for (int h = g; h < 2 * PAD_H; h += ng) {
            const int kp = h < PAD_H ? h : n + h;
            const float v = sl[mirror_fold(kp - PAD_H, n) * lb + l];
            for (int r = 0; r < nimg; ++r) col[size_t(kp) * a.pad_estride + size_t(images[r]) * a.pad_pitch] = v;
        }
    }
    // the x halo's columns whose source lies in this block, and the zeros
    // that fill the padded rows to their pitch (written by the last block)
    const int j = t & 31, w = t >> 5;
    const int xp = j < PAD_H ? j - PAD_H : nx + j - PAD_H;
    const int xs = mirror_fold(xp, nx) - xb;
    const bool hit = unsigned(xs) < unsigned(nl);
    const int xz = nx + 2 * PAD_H + j;
    const bool zero = xb + nl == nx && xz < a.pad_pitch;
    if (!__any_sync(0xffffffffu, hit || zero)) return;
    for (int kp = w; kp < np; kp += PF_NW) {
        const float v = hit ? sl[mirror_fold(kp - PAD_H, n) * lb + xs] : 0.0f;
        float *row = a.pad + size_t(kp) * a.pad_estride;
        for (int r = 0; r < nimg; ++r) {
            float *q = row + size_t(images[r]) * a.pad_pitch;
            if (hit) q[xp + PAD_H] = v;
            if (zero) q[xz] = 0.0f;
        }
    }
}

// lines per block: at most 32 and 64 KB of staged lines, fewer while the
// launch would have less than two blocks per SM (the recursion of the
// block's lines is its critical path)
static int lines_per_block(int n, int lines_total, int blocks_per_line_group)
{
    int lb = 32;
    while (lb > 1 && size_t(lb) * (n | 1) * sizeof(float) > 64 * 1024) lb >>= 1;
    const int nsm = device_sm_count();
    while (lb > 8 && size_t((lines_total + lb - 1) / lb) * blocks_per_line_group < size_t(2 * nsm)) lb >>= 1;
    return lb;
}

int prefilter_x_blocks(int dim, int nx, int ny, int nz)
{
    const int nlines = ny * (dim == 3 ? nz : 1);
    const int lb = lines_per_block(nx, nlines, 1);
    return (nlines + lb - 1) / lb;
}

void launch_prefilter(const float *src, float *coef, float *pad, int dim, int nx, int ny, int nz, float2 *mmpart,
                      unsigned *counter, float *minmax, cudaStream_t st)
{
    if (dim == 2) nz = 1;
    PrefilterPass a = {};
    a.in = src;
    a.out = coef;
    a.n = nx;
    a.nlines = ny * nz;
    a.lb = lines_per_block(nx, a.nlines, 1);
    a.mmpart = mmpart;
    a.counter = counter;
    a.minmax = minmax;
    size_t sm = size_t(a.lb) * (nx | 1) * sizeof(float);
    raise_smem_limit(reinterpret_cast<const void *>(k_prefilter_x), sm);
    k_prefilter_x<<<(a.nlines + a.lb - 1) / a.lb, PF_NT, sm, st>>>(a);
    count_launch();
    const size_t nxy = size_t(nx) * ny;
    for (int axis = 1; axis < dim; ++axis) {
        const bool last = axis == dim - 1;
        const int other = axis == 1 ? nz : ny;
        a.in = coef;
        a.n = axis == 1 ? ny : nz;
        a.nlines = nx;
        a.lb = lines_per_block(a.n, nx, other);
        a.estride = axis == 1 ? size_t(nx) : nxy;
        a.bstride = axis == 1 ? nxy : size_t(nx);
        sm = size_t(a.lb) * a.n * sizeof(float);
        const dim3 grid((nx + a.lb - 1) / a.lb, other);
        if (last) {
            a.pad = pad;
            a.pad_pitch = pad_pitch(nx);
            a.ny = dim == 3 ? ny : 0;
            a.pad_estride = dim == 3 ? size_t(a.pad_pitch) * (ny + 2 * PAD_H) : size_t(a.pad_pitch);
            raise_smem_limit(reinterpret_cast<const void *>(k_prefilter_cols<true>), sm);
            k_prefilter_cols<true><<<grid, PF_NT, sm, st>>>(a);
        } else {
            raise_smem_limit(reinterpret_cast<const void *>(k_prefilter_cols<false>), sm);
            k_prefilter_cols<false><<<grid, PF_NT, sm, st>>>(a);
        }
        count_launch();
    }
}

// The means of the two images in double (NCC provisional centres), and the
// copy of the reference into the level in the same pass.  Per-block partial
// sums in a fixed order, added by the last block.  FP64 instructions bound
// it (two additions per voxel at 1/64 of the FP32 rate), so values are widened
// beside that pipe (widen).
__global__ void __launch_bounds__(256) k_image_means(const float *__restrict__ src, const float *__restrict__ ref,
                                                     float *__restrict__ ref_out, size_t n, double *part,
                                                     unsigned *counter, double *out)
{
    __shared__ double red[16];
    __shared__ bool last;
    double v[2] = {0.0, 0.0};
    const size_t step = size_t(gridDim.x) * 256;
    for (size_t i0 = blockIdx.x * size_t(256) + threadIdx.x; i0 < n; i0 += 4 * step) {
        float a[4], b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const size_t i = i0 + j * step;
            a[j] = i < n ? __ldg(src + i) : 0.0f;
            b[j] = i < n ? __ldcg(ref + i) : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const size_t i = i0 + j * step;
            if (i < n) {
                v[0] += widen(a[j]);
                v[1] += widen(b[j]);
                if (ref_out) ref_out[i] = b[j];
            }
        }
    }
    block_sum<2>(v, red);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = v[0];
        part[gridDim.x + blockIdx.x] = v[1];
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    v[0] = v[1] = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += 256) {
        v[0] += __ldcg(part + i);
        v[1] += __ldcg(part + gridDim.x + i);
    }
    block_sum<2>(v, red);
    if (threadIdx.x == 0) {
        out[0] = v[0] / double(n);
        out[1] = v[1] / double(n);
        *counter = 0;
    }
}

void launch_image_means(const float *src, const float *ref, float *ref_out, size_t n, double *part, unsigned *counter,
                        double *out, cudaStream_t st)
{
    const int nb = int(std::min<size_t>(1024, (n + 255) / 256));
    k_image_means<<<nb, 256, 0, st>>>(src, ref, ref_out, n, part, counter, out);
    count_launch();
}

bool encode_pad_tmap(CUtensorMap *map, const float *pad, int nx, int ny, int nz)
{
    // resolved once, thread-safe (levels are made on several host threads)
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
        return PFN_cuTensorMapEncodeTiled_v12000(nullptr);
    }();
    if (!fn) return false;
    const int P = pad_pitch(nx);
    const cuuint64_t dims[3] = {cuuint64_t(P), cuuint64_t(ny + 2 * PAD_H), cuuint64_t(nz + 2 * PAD_H)};
    const cuuint64_t strides[2] = {cuuint64_t(P) * 4, cuuint64_t(P) * (ny + 2 * PAD_H) * 4};
    const cuuint32_t box[3] = {64, 16, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(pad), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

size_t pad_floats(int dim, int nx, int ny, int nz)
{
    const int planes = dim == 3 ? nz + 2 * PAD_H : 1;
    return size_t(pad_pitch(nx)) * (ny + 2 * PAD_H) * planes;
}

}  // namespace mgr
