// mgr_cost.cuh — cost finalisation shared by the split and plain paths.
#pragma once

#include "mgr_common.cuh"
#include "mgr_kernels.hh"

namespace mgr {

// Final SSD / NCC cost and force constants from the reduced sums, by the lanes
// of one warp (all call it with the same sums; lane 0 writes them, and has
// the value and the force pass' cost in the returned pair).  SSD: s[0] =
// sum (a-b)^2; value 0.5*s (x 1/N with norm) as FEvalSSD
// (mia/template/ssd.hh:54-99).  NCC: s = sums of da = a - c_a, db = b - c_b,
// da^2, db^2, da*db about provisional centres; value and gradient helper as
// NCCSums::value / get_grad_helper of the SSE2 build
// (mia/core/nccsum.cc:31-120: 1e-10 and 1e-5 thresholds).  The quotients that
// do not depend on one another are taken by different lanes: a division is a
// chain of FP64 instructions, the longest part of a finalisation.
__device__ __forceinline__ double2 finalise_cost(const EvalArgs &a, const double s[5], size_t N)
{
    const int lane = threadIdx.x & 31;
    double *sc = a.scalars;
    if (a.cost == 0) {
        const double scale = a.ssd_norm ? 0.5 / double(N) : 0.5, value = scale * s[0];
        if (lane != 0) return make_double2(value, value);
        sc[SC_VALUE] = value;
        sc[SC_FORCE_COST] = value;
        sc[SC_FSCALE] = a.ssd_norm ? double(float(1.0 / double(N))) : 1.0;
        sc[SC_K1] = sc[SC_K2] = sc[SC_MA] = sc[SC_MB] = 0.0;
        return make_double2(value, value);
    }
    const double n = double(N);
    const double sa = s[0], sb = s[1], saa = s[2], sbb = s[3], sab = s[4];
    const double ca = a.centers[0], cb = a.centers[1];
    const double num = lane == 0 ? sa : lane == 1 ? sb : lane == 2 ? sa * sa : lane == 3 ? sb * sb : sa * sb;
    const double q = num / n;
    auto quotient = [](double x, int from) { return __shfl_sync(0xffffffffu, x, from); };
    const double ma = ca + quotient(q, 0), mb = cb + quotient(q, 1);
    const double s2a = saa - quotient(q, 2);
    const double s2b = sbb - quotient(q, 3);
    const double cab = sab - quotient(q, 4);
    const double p1 = s2a * s2b;
    const double r = (lane == 0 ? cab * cab : cab) / (lane == 2 ? s2a : p1);
    const double r0 = quotient(r, 0), r1 = quotient(r, 1), r2 = quotient(r, 2);   // cab^2 / p1, cab / p1, cab / s2a
    double v = 1.0;
    if (p1 > 1e-10) v = 1.0 - r0;
    else if (s2a < 1e-5 && s2b < 1e-5) v = 0.0;
    double fv = 1.0, k1 = 0.0, k2 = 0.0, hma = 0.0, hmb = 0.0;
    if (p1 > 1e-5) {
        fv = 1.0 - r0;
        k1 = 2.0 * r1;
        k2 = r2;
        hma = ma;
        hmb = mb;
    } else if (s2a < 1e-5 && s2b < 1e-5) {
        fv = 0.0;
    }
    if (lane != 0) return make_double2(v, fv);
    sc[SC_VALUE] = v;
    sc[SC_FORCE_COST] = fv;
    sc[SC_K1] = k1;
    sc[SC_K2] = k2;
    sc[SC_MA] = hma;
    sc[SC_MB] = hmb;
    sc[SC_FSCALE] = 1.0;
    return make_double2(v, fv);
}

// Reduce the per-tile sums in a fixed order (every thread of the last block
// calls this, NT threads), then finalise the cost.
template <int NT = 256>
__device__ __forceinline__ void reduce_tile_sums(const EvalArgs &a, int ntiles, size_t N, double *red)
{
    double v[5] = {0, 0, 0, 0, 0};
    if (a.cost != 0) {
        strided_sums<4>(a.tile_sums, ntiles, threadIdx.x, NT, 5, v);
        block_sum<5, NT / 32>(v, red);
    } else {
        double v1[1] = {0.0};
        strided_sums<8>(a.tile_sums, ntiles, threadIdx.x, NT, 5, v1);
        block_sum<1, NT / 32>(v1, red);
        v[0] = v1[0];
    }
    if (threadIdx.x < 32) finalise_cost(a, v, N);
}

// The last block: a deferred SSD cost from the warp kernel's tile sums (the
// order of reduce_tile_sums), the blocks' penalty shares, the weighted costs.
// force: the image cost is the force pass', not the value's.  NT threads.
template <int NT>
__device__ __forceinline__ void gather_costs(const EvalArgs &a, int ntiles, int nblk, bool force, size_t N, double *red)
{
    const int tid = threadIdx.x;
    const bool fin = a.defer_cost && a.cost == 0;
    double *sc = a.scalars;
    double im = 0.0;
    unsigned flags[2] = {0u, 0u};
    if (tid == 0) {
        if (!fin) im = __ldcg(sc + (force ? SC_FORCE_COST : SC_VALUE));
        if (a.host_out) {
            flags[0] = __ldcg(&a.counters[6]);
            flags[1] = __ldcg(&a.counters[7]);
        }
    }
    // the first elements of both sums in flight together
    constexpr int B = 4;
    double x[B], y[B], vt[1] = {0.0}, vp[1] = {0.0};
#pragma unroll
    for (int j = 0; j < B; ++j) {
        const int t = tid + j * NT;
        x[j] = fin && t < ntiles ? __ldcg(a.tile_sums + size_t(t) * 5) : 0.0;
        y[j] = t < nblk ? __ldcg(a.pen_part + t) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < B; ++j) {
        const int t = tid + j * NT;
        if (fin && t < ntiles) vt[0] += x[j];
        if (t < nblk) vp[0] += y[j];
    }
    if (fin) strided_sums<8>(a.tile_sums, ntiles, tid + B * NT, NT, 5, vt);
    strided_sums<8>(a.pen_part, nblk, tid + B * NT, NT, 1, vp);
    double v2[2] = {vt[0], vp[0]};
    block_sum<2, NT / 32>(v2, red);
    if (tid >= 32) return;
    if (fin) {
        const double s5[5] = {v2[0], 0.0, 0.0, 0.0, 0.0};
        const double2 v = finalise_cost(a, s5, N);
        im = force ? v.y : v.x;
    }
    if (tid != 0) return;
    const double pen = a.has_penalty ? v2[1] : 0.0;
    const double ci = a.cost_weight * im, cp = a.has_penalty ? a.pen_weight * pen : 0.0;
    sc[SC_PEN] = pen;
    sc[SC_COST_IMG] = ci;
    sc[SC_COST_PEN] = cp;
    if (a.costs) {
        a.costs[0] = ci;
        a.costs[1] = cp;
    }
    if (a.host_out) {
        // the costs and both status flags to the caller's host memory; the
        // non-finite flag is cleared for the next call (every block has read
        // it before its arrival)
        a.host_out[0] = ci;
        a.host_out[1] = cp;
        unsigned *hf = reinterpret_cast<unsigned *>(a.host_out + 2);
        hf[0] = flags[0];
        hf[1] = flags[1];
        a.counters[7] = 0;
    }
    a.counters[1] = 0;
}

__device__ __forceinline__ float aw_at(const float4 *aw, int i, int k)
{
    return reinterpret_cast<const float *>(aw)[i * 4 + k];
}

}  // namespace mgr
