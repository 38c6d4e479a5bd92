// split.cu — the split evaluation path (default).  3D runs the z-walking
// kernels of split3.cu; the 2D kernels are here:
//
//   k_warp2<TX,TY>     per pixel tile: the tile's coefficient footprint is
//       contracted along y, then x (C2DSplineTransformation, on_grid,
//       mia/2d/transform/spline.cc:640-666) to the displacement u(x); the
//       prefiltered moving image is sampled with the bicubic B-spline at
//       x - u(x) (mia/2d/interpolator.cxx:216-311, mirror boundary, clamp);
//       the warped image is written and the SSD / NCC sums accumulated.
//   k_adjoint2<TX,TY>  per pixel tile: central differences of the warped
//       image (mia/2d/image.cc:351-391), the SSD / NCC force
//       (mia/template/ssd.hh:126-181), and the transposed spline contraction
//       (translate, mia/2d/transform/spline.cc:540-576) of the force onto
//       the tile's coefficient footprint, x then y; the result goes to the
//       tile's partial slot (no atomics).
//
// The per-coefficient gather of the partial slots and the divcurl penalty
// follow in gather.cu.
//
// 2D problems are small (frames of 96x96 to 1024x1024): the length of each
// kernel's chain of dependent steps bounds them, not a throughput.  So the
// kernels are launched to overlap (pdl_wait), load everything that does not
// depend on the kernel before them ahead of that wait, take the taps from
// global memory (one round of 16 independent loads; staging them in shared
// memory costs two more barriers and a copy).  1024x1024 NCC (1024 tiles) is
// the other end: there the warp kernel's FP64 sums and the adjoint kernel's
// shared-memory reads were the time; with four threads per sum, component
// pairs and whole lines per thread 26 -> 22 and 15.7 -> 11.6 us, evaluations
// one after another 26.6 -> 21.9 us (96x96 SSD 30.7 -> 30.1); the adjoint's
// voxel ranges from a table instead of two dependent loads 21.8 -> 21.4 us.
#include "mgr_cost.cuh"
#include "mgr_launch.hh"

namespace mgr {

namespace {

constexpr int NT = 256;
constexpr int ACC_P = 36;   // pitch of a warp's 32 values (banks four apart from warp to warp)
// resident blocks per SM of the warp kernel, whose threads wait for their
// taps most of the time: 1024x1024 NCC 24.7 us an evaluation with the
// compiler's choice, 21.9 with 4, 23.1 with 6, 24.1 with 8 (spills)
constexpr int WARP2_MINB = 4;

// bicubic sample at (px, py): from the mirror-padded copy while the taps lie
// inside it, else with the indices folded on the unpadded image (sample2);
// the same weights and summation order
__device__ __forceinline__ float taps2(const EvalArgs &a, float px, float py, float mn, float mx)
{
    const int nx = a.n[0], ny = a.n[1];
    const int fx = ffloor16(px), fy = ffloor16(py);
    const int sx = fx - 1, sy = fy - 1;
    constexpr int H = PAD_H;
    if (sx >= -H && sx + 3 < nx + H && sy >= -H && sy + 3 < ny + H) {
        const int P = pad_pitch(nx);
        return sample2_at(a.coef_pad + size_t(sy + H) * P + (sx + H), P, px, py, fx, fy, mn, mx);
    }
    return sample2(a.coef_img, nx, ny, px, py, mn, mx);
}

}  // namespace

// ---------------------------------------------------------------------
// warp
// ---------------------------------------------------------------------
// tile (bx, by) of a pair with `ntiles` tiles, `tile` its linear index.  A
// thread keeps its x column and takes every (NT / TX)-th row of the tile.
template <int TX, int TY>
__device__ __forceinline__ void warp2_body(const EvalArgs &a, int bx, int by, int ntiles, int tile)
{
    static_assert(NT % TX == 0 && TY % (NT / TX) == 0, "every thread has its column and whole rows");
    constexpr int NR = NT / TX, PT = TY / NR;
    extern __shared__ __align__(16) float sm[];
    __shared__ double red[5 * (NT / 32)];
    __shared__ float accs[5][(NT / 32) * ACC_P];
    __shared__ float csc[2];   // NCC centres (converted once per block)
    __shared__ int fsy[TY];
    __shared__ float4 fwy[TY];
    __shared__ bool is_last;
    const Axis &X = a.ax[0], &Y = a.ax[1];
    const int nx = a.n[0], ny = a.n[1];
    const int x0 = bx * TX, y0 = by * TY;
    const int FX = X.fc, FY = Y.fc;
    const int cx0 = X.ftile0[bx], cy0 = Y.ftile0[by];
    const int ncx = a.nc[0], ncy = a.nc[1];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    float *C = sm;                  // [2][FY][FX]
    float *T2 = C + 2 * FY * FX;    // [2][TY][FX]

    // the level's tables and images, ahead of the wait
    const int xx = tid % TX, yy0 = tid / TX;
    const int x = x0 + xx, xc = min(x, nx - 1);
    const int s = X.fs[xc] - cx0;
    const float4 w = X.fw[xc];
    if (tid < TY) {
        const int y = min(y0 + tid, ny - 1);
        fsy[tid] = Y.fs[y] - cy0;
        fwy[tid] = Y.fw[y];
    }
    float b[PT];
#pragma unroll
    for (int k = 0; k < PT; ++k) {
        const int y = y0 + yy0 + k * NR;
        b[k] = x < nx && y < ny ? __ldg(a.ref + size_t(y) * nx + x) : 0.0f;
    }
    const float mn = a.minmax[0], mxv = a.minmax[1];
    if (tid < 2) csc[tid] = a.cost == 0 ? 0.0f : float(a.centers[tid]);

    pdl_wait();
    pdl_trigger();
    // coefficient footprint: rows iy of 2 FX consecutive values (parameters
    // are interleaved per node).  A single evaluation reads the caller's
    // doubles, on the device or in host memory, where a non-finite value is
    // taken as 0 and flagged; the blocks write the float copy that the
    // gather reads between them.
    const double *const src = a.params_host ? a.params_host : a.params;
    bool nonfinite = false;
    auto param = [&](size_t i) -> float {
        if (!a.convert) return a.params_f[i];
        const double v = src[i];
        if (a.params_host && !isfinite(v)) {
            nonfinite = true;
            return 0.0f;
        }
        return float(v);
    };
    const int w2 = 2 * FX;
    for (int e = tid; e < FY * w2; e += NT) {
        const int iy = e / w2, j = e - iy * w2;
        float v = 0.0f;
        if (cx0 + (j >> 1) < ncx && cy0 + iy < ncy) v = param((size_t(cy0 + iy) * ncx + cx0) * 2 + j);
        C[((j & 1) * FY + iy) * FX + (j >> 1)] = v;
    }
    if (a.convert) {
        const size_t n = size_t(ncx) * ncy * 2, per = (n + ntiles - 1) / ntiles;
        const size_t i1 = min(n, per * (tile + 1));
        for (size_t i = per * tile + tid; i < i1; i += NT) a.params_f[i] = param(i);
        if (nonfinite) atomicOr(&a.counters[7], 1u);
    }
    __syncthreads();
    // y stage
    for (int e = tid; e < 2 * TY * FX; e += NT) {
        const int r = e / FX, ix = e - r * FX;
        const int yy = r % TY;
        const float4 wy = fwy[yy];
        const float *c = C + ((r / TY) * FY + fsy[yy]) * FX + ix;
        T2[e] = wy.x * c[0] + wy.y * c[FX] + wy.z * c[2 * FX] + wy.w * c[3 * FX];
    }
    __syncthreads();

    // x stage, bicubic sample, warped image, sums
    float acc[5] = {0, 0, 0, 0, 0};
    const float ca = csc[0], cb = csc[1];
#pragma unroll
    for (int k = 0; k < PT; ++k) {
        const int yy = yy0 + k * NR, y = y0 + yy;
        if (x >= nx || y >= ny) continue;
        float p[2];
#pragma unroll
        for (int comp = 0; comp < 2; ++comp) {
            const float *c = T2 + (comp * TY + yy) * FX + s;
            const float u = w.x * c[0] + w.y * c[1] + w.z * c[2] + w.w * c[3];
            p[comp] = float(comp == 0 ? x : y) - u;
        }
        const float wv = taps2(a, p[0], p[1], mn, mxv);
        a.warped[size_t(y) * nx + x] = wv;
        if (a.cost == 0) {
            const float d = wv - b[k];
            acc[0] += d * d;
        } else {
            const float da = wv - ca, db = b[k] - cb;
            acc[0] += da;
            acc[1] += db;
            acc[2] += da * da;
            acc[3] += db * db;
            acc[4] += da * db;
        }
    }
    // tile sums: per warp warp_sum's tree over its 32 lanes in double, then a
    // tree over the eight warps.  FP64 additions are the kernel's slowest
    // instructions (five trees by every lane took half of it at 1024x1024),
    // so the values go through shared memory and four threads sum a tree: the
    // lanes j, j + 4, ... of a warp each (levels 16, 8, 4), then among
    // themselves (levels 2, 1).
    constexpr int NW = NT / 32;
    static_assert(NW == 8, "the tree over the warps");
    const int ncomp = a.cost == 0 ? 1 : 5;
#pragma unroll
    for (int k = 0; k < 5; ++k)
        if (k < ncomp) accs[k][wid * ACC_P + lane] = acc[k];
    __syncthreads();
    if (tid < ncomp * 32) {
        const int k = tid >> 5, w8 = (tid >> 2) & 7, j = tid & 3;
        const float *f = &accs[k][w8 * ACC_P + j];
        double t[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) t[m] = widen(f[4 * m]) + widen(f[4 * m + 16]);
        double v = (t[0] + t[2]) + (t[1] + t[3]);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        if (j == 0) red[k * NW + w8] = v;
    }
    __syncthreads();
    if (tid < 5) {
        double v = 0.0;
        if (tid == 0 || a.cost != 0) {
            const double *r = red + tid * NW;
            v = ((r[0] + r[4]) + (r[2] + r[6])) + ((r[1] + r[5]) + (r[3] + r[7]));
        }
        a.tile_sums[size_t(tile) * 5 + tid] = v;
    }
    // a deferred finalisation (SSD: the gather's last block) needs no
    // last-block pass here
    if (a.defer_cost) return;
    __syncthreads();
    if (tid == 0) is_last = arrive_last(&a.counters[0], ntiles);
    __syncthreads();
    if (is_last) {
        reduce_tile_sums(a, ntiles, size_t(nx) * ny, red);
        if (tid == 0) a.counters[0] = 0;
    }
}

// ---------------------------------------------------------------------
// gradient + force + adjoint
// ---------------------------------------------------------------------
template <int TX, int TY>
__device__ __forceinline__ void adjoint2_body(const EvalArgs &a, int bx, int by, int tile_index)
{
    constexpr int NR = NT / TX, PT = TY / NR, TXP = TX + 1;
    // the x stage by whole lines or by outputs (below)
    constexpr bool LINES = TY >= 16;
    extern __shared__ __align__(16) float sm[];
    __shared__ int asx[TX], asy[TY];
    __shared__ float awx[TX * 4], awy[TY * 4];
    __shared__ float4 awx2[LINES ? TX : 1][2];   // LINES: awx, each weight twice
    __shared__ float fsc[5];   // force constants (converted once per block)
    const Axis &X = a.ax[0], &Y = a.ax[1];
    const int nx = a.n[0], ny = a.n[1];
    const int x0 = bx * TX, y0 = by * TY;
    const int ex = min(TX, nx - x0), ey = min(TY, ny - y0);
    const int AXc = X.ac, AYc = Y.ac;
    const int ax0 = X.atile0[bx], ay0 = Y.atile0[by];
    const int tid = threadIdx.x, lane = tid & 31;
    float *part = a.partial + size_t(tile_index) * a.slot;
    // both components side by side: their arithmetic runs on register pairs
    float2x *F = reinterpret_cast<float2x *>(sm);         // [TY][TXP]
    float2x *AX = F + TY * TXP;                           // [TY][AXc]
    int2 *rx = reinterpret_cast<int2 *>(AX + TY * AXc);   // [AXc] columns of a coefficient
    int2 *ry = rx + AXc;                                  // [AYc] rows

    // the level's tables and the reference, ahead of the wait
    for (int e = tid; e < TX * 4; e += NT) {
        const int xc = min(x0 + e / 4, nx - 1);
        awx[e] = reinterpret_cast<const float *>(X.aw)[size_t(xc) * 4 + (e & 3)];
        if (LINES) reinterpret_cast<float2 *>(awx2[e / 4])[e & 3] = make_float2(awx[e], awx[e]);
        if ((e & 3) == 0) asx[e / 4] = X.as[xc] - ax0;
    }
    for (int e = tid; e < TY * 4; e += NT) {
        const int yc = min(y0 + e / 4, ny - 1);
        awy[e] = reinterpret_cast<const float *>(Y.aw)[size_t(yc) * 4 + (e & 3)];
        if ((e & 3) == 0) asy[e / 4] = Y.as[yc] - ay0;
    }
    // the tile's voxels whose four coefficients include one (none beyond the
    // grid)
    for (int o = tid; o < AXc + AYc; o += NT) {
        const bool isx = o < AXc;
        const Axis &A = isx ? X : Y;
        const int c = isx ? ax0 + o : ay0 + o - AXc, v0 = isx ? x0 : y0, e = isx ? ex : ey;
        const int2 r = c < A.nc ? A.win[c] : make_int2(0, 0);
        rx[o] = make_int2(max(r.x - v0, 0), min(r.y - v0, e));
    }
    const int xx = tid % TX, yy0 = tid / TX;
    const int x = x0 + xx;
    float b[PT];
#pragma unroll
    for (int k = 0; k < PT; ++k) {
        const int y = y0 + yy0 + k * NR;
        b[k] = x < nx && y < ny ? __ldg(a.ref + size_t(y) * nx + x) : 0.0f;
    }
    // the warped image and the cost's scalars come from the warp kernel
    pdl_wait();
    pdl_trigger();
    if (tid < 5) {
        // the SSD force scale from the settings, as the finalisation sets it
        // (with a deferred finalisation it is not set yet)
        if (a.cost != 0) fsc[tid] = float(a.scalars[SC_K1 + tid]);
        else if (tid == 4) fsc[4] = a.ssd_norm ? float(1.0 / double(size_t(nx) * ny)) : 1.0f;
    }
    // (a lane's x neighbours are the lanes beside it: TX is a multiple of 32)
    float wc[PT], wl[PT], wr[PT], wu[PT], wd[PT];
#pragma unroll
    for (int k = 0; k < PT; ++k) {
        const int y = y0 + yy0 + k * NR;
        const bool in = x < nx && y < ny;
        const float *p = a.warped + (in ? size_t(y) * nx + x : 0);
        wc[k] = in ? __ldcg(p) : 0.0f;
        wu[k] = in && y > 0 ? __ldcg(p - nx) : 0.0f;
        wd[k] = in && y < ny - 1 ? __ldcg(p + nx) : 0.0f;
        wl[k] = in && lane == 0 && x > 0 ? __ldcg(p - 1) : 0.0f;
        wr[k] = in && lane == 31 && x < nx - 1 ? __ldcg(p + 1) : 0.0f;
    }
    __syncthreads();
    {
        const float k1 = fsc[0], k2 = fsc[1], ma = fsc[2], mb = fsc[3], fscale = fsc[4];
#pragma unroll
        for (int k = 0; k < PT; ++k) {
            const int yy = yy0 + k * NR, y = y0 + yy;
            float left = __shfl_up_sync(0xffffffffu, wc[k], 1), right = __shfl_down_sync(0xffffffffu, wc[k], 1);
            if (lane == 0) left = wl[k];
            if (lane == 31) right = wr[k];
            float f[2] = {0.0f, 0.0f};
            if (x < nx && y < ny) {
                const float w = wc[k];
                float g[2];
                g[0] = (x > 0 && x < nx - 1) ? 0.5f * (right - left) : 0.0f;
                g[1] = (y > 0 && y < ny - 1) ? 0.5f * (wd[k] - wu[k]) : 0.0f;
                if (a.cost == 0) {
                    const float d = w - b[k];
                    f[0] = (g[0] * d) * fscale;
                    f[1] = (g[1] * d) * fscale;
                } else {
                    const float s = k1 * (k2 * (w - ma) - (b[k] - mb));
                    f[0] = s * g[0];
                    f[1] = s * g[1];
                }
            }
            F[yy * TXP + xx] = pack2(f[0], f[1]);
        }
    }
    __syncthreads();
    // x stage.  Tall tiles: a thread per row, a sliding window of four sums
    // over its columns (a third of the loads, and shared-memory reads bound
    // the kernel where there are many tiles); flat ones, of small images: a
    // thread per output, the output's columns ascending (a short chain, all
    // threads busy).  The same sums.
    if (LINES) {
        if (tid < ey) {
            const float2x *f = F + tid * TXP;
            float2x *dst = AX + tid * AXc;
            float2x s0 = 0, s1 = 0, s2 = 0, s3 = 0;
            int oc = 0;
#pragma unroll 4
            for (int i = 0; i < ex; ++i) {
                const int o = asx[i];
                while (oc < o) {
                    dst[oc] = s0;
                    s0 = s1;
                    s1 = s2;
                    s2 = s3;
                    s3 = 0;
                    ++oc;
                }
                const float4 u = awx2[i][0], v = awx2[i][1];
                const float2x g = f[i];
                s0 = fma2(pack2(u.x, u.y), g, s0);
                s1 = fma2(pack2(u.z, u.w), g, s1);
                s2 = fma2(pack2(v.x, v.y), g, s2);
                s3 = fma2(pack2(v.z, v.w), g, s3);
            }
            if (oc < AXc) dst[oc] = s0;
            if (oc + 1 < AXc) dst[oc + 1] = s1;
            if (oc + 2 < AXc) dst[oc + 2] = s2;
            if (oc + 3 < AXc) dst[oc + 3] = s3;
            for (int o = oc + 4; o < AXc; ++o) dst[o] = 0;
        }
    } else {
        for (int e = tid; e < ey * AXc; e += NT) {
            const int r = e / AXc, ox = e - r * AXc;
            const float2x *f = F + r * TXP;
            const int2 v = rx[ox];
            float2x acc = 0;
#pragma unroll 4
            for (int i = v.x; i < v.y; ++i) {
                const float w = awx[i * 4 + (ox - asx[i])];
                acc = fma2(pack2(w, w), f[i], acc);
            }
            AX[e] = acc;
        }
    }
    __syncthreads();
    // y stage: coefficient (oy, ox), its rows ascending, into the slot
    for (int e = tid; e < AYc * AXc; e += NT) {
        const int oy = e / AXc, ox = e - oy * AXc;
        const float2x *f = AX + ox;
        const int2 v = ry[oy];
        float2x acc = 0;
#pragma unroll 4
        for (int i = v.x; i < v.y; ++i) {
            const float w = awy[i * 4 + (oy - asy[i])];
            acc = fma2(pack2(w, w), f[i * AXc], acc);
        }
        reinterpret_cast<float2x *>(part)[e] = acc;
    }
}

// ---------------------------------------------------------------------
// kernels: one pair (grid = tiles) and a batch of pairs (grid = work list
// of (pair, tile) items; pairs whose minimizer has finished are skipped)
// ---------------------------------------------------------------------
template <int TX, int TY>
__global__ void __launch_bounds__(NT, WARP2_MINB) k_warp2(const __grid_constant__ EvalArgs a)
{
    warp2_body<TX, TY>(a, blockIdx.x, blockIdx.y, gridDim.x * gridDim.y, blockIdx.y * gridDim.x + blockIdx.x);
}

template <int TX, int TY>
__global__ void __launch_bounds__(NT) k_adjoint2(const __grid_constant__ EvalArgs a)
{
    adjoint2_body<TX, TY>(a, blockIdx.x, blockIdx.y, blockIdx.y * gridDim.x + blockIdx.x);
}

template <int TX, int TY>
__global__ void __launch_bounds__(NT, WARP2_MINB) k_warp2_batch(const EvalArgs *__restrict__ args, const int2 *__restrict__ items,
                                                    const int *__restrict__ active)
{
    const int2 it = items[blockIdx.x];
    pdl_wait();   // the minimizer sets the flags
    if (!active[it.x]) return;
    const EvalArgs &a = args[it.x];
    const int ntx = a.ax[0].nt;
    warp2_body<TX, TY>(a, it.y % ntx, it.y / ntx, ntx * a.ax[1].nt, it.y);
}

template <int TX, int TY>
__global__ void __launch_bounds__(NT) k_adjoint2_batch(const EvalArgs *__restrict__ args,
                                                       const int2 *__restrict__ items, const int *__restrict__ active)
{
    const int2 it = items[blockIdx.x];
    pdl_wait();   // the minimizer sets the flags
    if (!active[it.x]) return;
    const EvalArgs &a = args[it.x];
    const int ntx = a.ax[0].nt;
    adjoint2_body<TX, TY>(a, it.y % ntx, it.y / ntx, it.y);
}

// ---------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------
static size_t warp_smem(const EvalArgs &a)
{
    const Axis &X = a.ax[0], &Y = a.ax[1];
    return size_t(2) * (Y.fc + Y.t) * X.fc * sizeof(float);
}

static size_t adjoint_smem(const EvalArgs &a)
{
    const Axis &X = a.ax[0], &Y = a.ax[1];
    return (size_t(2) * Y.t * (X.t + 1 + X.ac) + 2 * (X.ac + Y.ac)) * sizeof(float);
}

template <int TX, int TY>
static void launch_tile(const EvalArgs &a, int which, cudaStream_t st)
{
    const dim3 grid(a.ax[0].nt, a.ax[1].nt);
    if (which == 0) {
        const size_t sm = warp_smem(a);
        raise_smem_limit(reinterpret_cast<const void *>(k_warp2<TX, TY>), sm);
        // the first kernel of an evaluation: after everything queued before
        launch_pdl(false, k_warp2<TX, TY>, grid, dim3(NT), sm, st, a);
    } else {
        const size_t sm = adjoint_smem(a);
        raise_smem_limit(reinterpret_cast<const void *>(k_adjoint2<TX, TY>), sm);
        launch_pdl(a.pdl != 0, k_adjoint2<TX, TY>, grid, dim3(NT), sm, st, a);
    }
    count_launch();
}

// the 2D tile shapes compiled in (tile_supported() must match); 3D runs
// the z-walking kernels of split3.cu
static bool dispatch(const EvalArgs &a, int which, cudaStream_t st)
{
    if (a.dim == 3) {
        if (which == 0)
            launch_warp3(a, st);
        else
            launch_adjoint3(a, st);
        return true;
    }
    const int tx = a.ax[0].t, ty = a.ax[1].t;
#define MGR_TILE2(X_, Y_)                                  \
    if (tx == X_ && ty == Y_) {                            \
        launch_tile<X_, Y_>(a, which, st);           \
        return true;                                       \
    }
    MGR_TILE2(32, 8)
    MGR_TILE2(32, 16)
    MGR_TILE2(64, 8)
    MGR_TILE2(64, 16)
    MGR_TILE2(32, 32)
#undef MGR_TILE2
    return false;
}

bool tile_supported(int dim, int tx, int ty, int tz)
{
    static const int t2[][2] = {{32, 8}, {32, 16}, {64, 8}, {64, 16}, {32, 32}};
    if (dim == 3) return tile_supported3(tx, ty, tz);
    for (auto &t : t2)
        if (t[0] == tx && t[1] == ty) return true;
    return false;
}

void launch_warp(const EvalArgs &a, cudaStream_t st)
{
    dispatch(a, 0, st);
}

void launch_adjoint(const EvalArgs &a, cudaStream_t st)
{
    dispatch(a, 1, st);
}

size_t split_smem(const EvalArgs &a, int which)
{
    if (a.dim == 3) return split3_smem(a, which);
    return which == 0 ? warp_smem(a) : adjoint_smem(a);
}

template <int TX, int TY>
static void launch_batch_tile(const EvalArgs *args, const int2 *items, int nitems, const int *active,
                              size_t sm, int which, bool pdl, cudaStream_t st)
{
    launch_pdl(pdl, which == 0 ? k_warp2_batch<TX, TY> : k_adjoint2_batch<TX, TY>, dim3(nitems), dim3(NT), sm, st, args,
               items, active);
    count_launch();
}

template <int TX, int TY>
static void prepare_batch_tile(size_t sm_warp, size_t sm_adj)
{
    // (only ever raised: another thread's batch may be running with more)
    raise_smem_limit(reinterpret_cast<const void *>(k_warp2_batch<TX, TY>), sm_warp);
    raise_smem_limit(reinterpret_cast<const void *>(k_adjoint2_batch<TX, TY>), sm_adj);
}

void prepare_split_batch(int dim, int cost, int tx, int ty, int tz, size_t sm_warp, size_t sm_adj)
{
    if (dim == 3) {
        if (tile_supported3_batch(tx, ty, tz)) prepare_split3_batch(cost, sm_warp, sm_adj);
        return;
    }
#define MGR_PTILE2(X_, Y_) \
    if (tx == X_ && ty == Y_) prepare_batch_tile<X_, Y_>(sm_warp, sm_adj);
    MGR_PTILE2(32, 8)
    MGR_PTILE2(32, 16)
    MGR_PTILE2(64, 8)
    MGR_PTILE2(64, 16)
    MGR_PTILE2(32, 32)
#undef MGR_PTILE2
}

bool launch_split_batch(int dim, int cost, int tx, int ty, int tz, const EvalArgs *args, const int2 *items, int nitems,
                        const int *active, size_t sm, int which, bool pdl, cudaStream_t st)
{
    if (dim == 3) {
        if (!tile_supported3_batch(tx, ty, tz)) return false;
        launch_split3_batch(cost, args, items, nitems, active, sm, which, pdl, st);
        return true;
    }
#define MGR_BTILE2(X_, Y_)                                                      \
    if (tx == X_ && ty == Y_) {                                                 \
        launch_batch_tile<X_, Y_>(args, items, nitems, active, sm, which, pdl, st); \
        return true;                                                            \
    }
    MGR_BTILE2(32, 8)
    MGR_BTILE2(32, 16)
    MGR_BTILE2(64, 8)
    MGR_BTILE2(64, 16)
    MGR_BTILE2(32, 32)
#undef MGR_BTILE2
    return false;
}

}  // namespace mgr
