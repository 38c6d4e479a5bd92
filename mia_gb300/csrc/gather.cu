// gather.cu — 2D: per-coefficient gather of the tile partials, the divcurl
// penalty (value and gradient) and the final weighted costs (3D: k_gather3 in
// split3.cu).
//
// One block owns 32 consecutive coefficients (lane = coefficient, so
// neighbour loads coalesce along x).  The eight warps split the work of
// those 32 coefficients: the cells of the boundary-clipped CSR row
// (mia/2d/ppmatrix.cc:328-352), and the partial slots of the split path that
// hold the coefficient.  The per-warp sums are combined in a fixed order
// (deterministic, no atomics), the penalty weight and sign
// (C3DSplineTransformPenalty::value_and_gradient,
// mia/3d/splinetransformpenalty.cc:60-71) and the full-cost weight
// (mia/template/fullcost.cxx:37-45) applied, and the last block finalises
// the costs.
//
// A few blocks with a chain of dependent loads (row range, cell, parameter;
// tile range, tile start, slot): latency bounds it, so the loads of a step
// are issued together and everything but the slots is done before the wait
// for the adjoint kernel.  Of 18.7 k cycles at 96x96 the last block's sums
// were 7 k and the blocks' ends 5 k: a warp per gradient component and one
// for the value, whose thread arrives with no other store in flight, and
// loads in flight together make it 10.3 -> 8.0 us (an evaluation from host
// memory 30.1 -> 28.7 us).
#include "mgr_cost.cuh"
#include "mgr_launch.hh"

namespace mgr {

namespace {
constexpr int GT = 256;   // threads per block
constexpr int GW = GT / 32;
constexpr int GC = 32;    // coefficients per block
constexpr int NPART = 7;  // per warp: penalty g[2], r[3]; image s[2]
constexpr int GCELLS = 7; // cells a warp loads at a time: a row has at most 49
constexpr int GSLOTS = 4; // partial slots a warp loads at a time
}  // namespace

// block `blk` of the pair's `nblk` gather blocks
__device__ __forceinline__ void gather2_body(const EvalArgs &a, int with_gradient, int image_from_dense, int blk,
                                             int nblk)
{
    __shared__ float part[GW][NPART][GC];
    __shared__ double red[2 * GW];
    __shared__ bool is_last;
    const Axis &X = a.ax[0], &Y = a.ax[1];
    const int ncx = a.nc[0], ncy = a.nc[1];
    const size_t ncoef = size_t(ncx) * ncy;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const size_t i = size_t(blk) * GC + lane;
    const bool valid = i < ncoef;
    const int cx = valid ? int(i % ncx) : 0;
    const int cy = valid ? int(i / ncx) : 0;

    // the first loads of both chains: the cells of the coefficient's row and
    // the slots that hold it (entries k = w, w + GW, ... of the tiles)
    const bool img = valid && with_gradient && !image_from_dense;
    const bool pen = valid && a.has_penalty;
    int nX = 0, nY = 0, e0 = 0, e1 = 0;
    if (img) {
        nX = X.glen[cx];
        nY = Y.glen[cy];
    }
    if (pen) {
        e0 = a.pen_rowptr[i] + w;
        e1 = a.pen_rowptr[i + 1];
    }
    const bool lists = nX >= 0 && nY >= 0;
    const int2 none = make_int2(0, -1);
    const int2 gx = img && !lists ? X.gtile[cx] : none, gy = img && !lists ? Y.gtile[cy] : none;
    if (!lists) {
        nX = gx.y - gx.x + 1;
        nY = gy.y - gy.x + 1;
    }
    const int total = (nX > 0 && nY > 0) ? nX * nY : 0;
    auto slot = [&](int k) -> const float * {
        const int jy = k / nX, jx = k - jy * nX;
        if (lists)
            return a.partial + (X.glist[size_t(cx) * GATHER_LMAX + jx] + Y.glist[size_t(cy) * GATHER_LMAX + jy]);
        const int tx = gx.x + jx, ty = gy.x + jy;
        const int lx = cx - X.atile0[tx], ly = cy - Y.atile0[ty];
        return a.partial + (size_t(ty) * X.nt + tx) * a.slot + (size_t(ly) * X.ac + lx) * 2;
    };
    // the second loads: cells, slot offsets
    float4 cell[GCELLS];
    int col[GCELLS];
    auto cells = [&]() {
#pragma unroll
        for (int u = 0; u < GCELLS; ++u) {
            const bool in = e0 + u * GW < e1;
            col[u] = in ? a.pen_col[e0 + u * GW] : -1;
            cell[u] = in ? a.pen_val[e0 + u * GW] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    cells();
    const float *sp[GSLOTS];
#pragma unroll
    for (int u = 0; u < GSLOTS; ++u) sp[u] = w + u * GW < total ? slot(w + u * GW) : nullptr;

    // The float copy of the parameters is complete before any block of this
    // kernel starts, except right after the warp kernel that makes it (the
    // value alone, no adjoint kernel between them); it is read through the
    // L2, never from a line an earlier kernel left in L1.
    if (!with_gradient) pdl_wait();
    float g[2] = {0.0f, 0.0f}, r[3] = {0, 0, 0}, s[2] = {0.0f, 0.0f};
    while (e0 < e1) {   // (at most once: a row has at most 49 cells)
        float2 c[GCELLS];
#pragma unroll
        for (int u = 0; u < GCELLS; ++u)
            c[u] = col[u] >= 0 ? __ldcg(reinterpret_cast<const float2 *>(a.params_f) + col[u])
                               : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int u = 0; u < GCELLS; ++u)
            if (col[u] >= 0) {
                const float cjx = c[u].x, cjy = c[u].y;
                const float4 v = cell[u];
                const float aa = cjx * v.x, bb = cjy * v.y, cxx = cjx * v.z, cyy = cjy * v.z;
                g[0] += aa + aa + cyy;
                g[1] += bb + bb + cxx;
                r[0] += aa;
                r[1] += cyy;
                r[2] += bb;
            }
        e0 += GW * GCELLS;
        if (e0 < e1) cells();
    }
    float2 ci = make_float2(0.0f, 0.0f);
    if (w == 2 && pen) ci = __ldcg(reinterpret_cast<const float2 *>(a.params_f) + i);
    if (with_gradient) pdl_wait();
    pdl_trigger();
    // parameters the warp kernel found non-finite: nothing is written to the
    // caller's buffers (read by every block before its arrival)
    const bool bad = a.params_host && *(volatile unsigned *)&a.counters[7] != 0u;
    {
        float2 v[GSLOTS];
#pragma unroll
        for (int u = 0; u < GSLOTS; ++u)
            v[u] = sp[u] ? __ldcg(reinterpret_cast<const float2 *>(sp[u])) : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int u = 0; u < GSLOTS; ++u)
            if (sp[u]) {
                s[0] += v[u].x;
                s[1] += v[u].y;
            }
    }
    for (int k = w + GSLOTS * GW; k < total; k += GW) {
        const float2 v = __ldcg(reinterpret_cast<const float2 *>(slot(k)));
        s[0] += v.x;
        s[1] += v.y;
    }
    part[w][0][lane] = g[0];
    part[w][1][lane] = g[1];
    part[w][2][lane] = r[0];
    part[w][3][lane] = r[1];
    part[w][4][lane] = r[2];
    part[w][5][lane] = s[0];
    part[w][6][lane] = s[1];
    __syncthreads();
    // the warps' sums of each quantity in warp order, quantity k by warp k
    if (w < NPART) {
        float t = 0.0f;
#pragma unroll
        for (int p = 0; p < GW; ++p) t += part[p][w][lane];
        part[0][w][lane] = t;
    }
    __syncthreads();
    // a warp per component of the gradient, one for the penalty's value and
    // the block's arrival
    if (w < 2) {
        if (valid && with_gradient && !bad) {
            const size_t o = i * 2 + w;
            const double gp = a.has_penalty ? a.pen_grad_w * widen(part[0][w][lane]) : 0.0;
            const double gi = image_from_dense ? a.grad_image[o] : a.cost_weight * widen(-part[0][5 + w][lane]);
            a.grad_total[o] = gi + gp;
            if (a.grad_image && !image_from_dense) a.grad_image[o] = gi;
            if (a.grad_penalty) a.grad_penalty[o] = gp;
        }
    } else if (w == 2) {
        double pval = 0.0;
        if (pen) pval = widen(ci.x * part[0][2][lane] + ci.x * part[0][3][lane] + ci.y * part[0][4][lane]);
        pval = warp_sum(pval);
        if (lane == 0) {
            a.pen_part[blk] = pval;
            is_last = arrive_last(&a.counters[1], nblk);
        }
    }
    __syncthreads();
    if (is_last) gather_costs<GT>(a, X.nt * Y.nt, nblk, with_gradient, size_t(a.n[0]) * a.n[1], red);
}

__global__ void __launch_bounds__(GT) k_gather2(const __grid_constant__ EvalArgs a, int with_gradient,
                                                int image_from_dense)
{
    gather2_body(a, with_gradient, image_from_dense, blockIdx.x, gridDim.x);
}

// batch: work list of (pair, block) items; finished pairs are skipped
__global__ void __launch_bounds__(GT) k_gather2_batch(const EvalArgs *__restrict__ args, const int2 *__restrict__ items,
                                                      const int *__restrict__ active, const int *__restrict__ nblocks)
{
    const int2 it = items[blockIdx.x];
    pdl_wait();   // the minimizer sets the flags
    if (!active[it.x]) return;
    gather2_body(args[it.x], 1, 0, it.y, nblocks[it.x]);
}

void launch_gather_batch(int dim, const EvalArgs *args, const int2 *items, int nitems, const int *active,
                         const int *nblocks, bool pdl, cudaStream_t st)
{
    if (dim == 3) {
        launch_gather3_batch(args, items, nitems, active, nblocks, pdl, st);
        return;
    }
    launch_pdl(pdl, k_gather2_batch, dim3(nitems), dim3(GT), 0, st, args, items, active, nblocks);
    count_launch();
}

int gather_blocks(const EvalArgs &a)
{
    if (a.dim == 3) return gather3_blocks(a);
    const size_t ncoef = size_t(a.nc[0]) * a.nc[1];
    return int((ncoef + GC - 1) / GC);
}

void launch_gather_mode(const EvalArgs &a, int with_gradient, int dense, cudaStream_t st)
{
    if (a.dim == 3) {
        launch_gather3(a, with_gradient, dense, st);
        return;
    }
    launch_pdl(a.pdl != 0, k_gather2, dim3(gather_blocks(a)), dim3(GT), 0, st, a, with_gradient, dense);
    count_launch();
}

void launch_gather(const EvalArgs &a, int with_gradient, cudaStream_t st)
{
    launch_gather_mode(a, with_gradient, 0, st);
}

}  // namespace mgr
