// split3.cu — the 3D split evaluation path.
//
// A tile is 32 (x) x 8 (y) x TZ (z) voxels; lane = x, warp = y (the adjoint
// kernel: two rows), and every thread walks its z column.  All threads of a
// block stand on the same z plane at the same step, so the z tables are
// uniform and the per-thread sliding windows below advance in lock step.
//
//   k_warp3<TZ>       the tile's coefficient footprint is contracted along x
//       and y in shared memory (C3DSplineTransformation::init_grid,
//       mia/3d/transform/spline.cc:541-653, x then y then z); each thread
//       keeps the four z coefficients of its column that the current voxel
//       needs in registers and slides them as z advances, giving u(x); the
//       prefiltered moving image is sampled with the tricubic B-spline at
//       x - u(x) (mia/3d/interpolator.cxx:250-287, mirror boundary, clamp
//       to [min(0, min src), max src]); the taps are read from a ring of z
//       planes in shared memory that bulk copies fill ahead of the walk from
//       a mirror-padded copy (the box of a plane follows from the range of
//       u over the tile), so the interior needs no index folding and the
//       gather costs shared-memory wavefronts instead of L1 lines; each
//       thread samples two planes per step (two independent tap chains in
//       flight); the warped image is written and the SSD / NCC sums are
//       accumulated (the cost is finalised after the kernel).
//   k_adjoint3<TZ>    central differences of the warped image (x and y
//       neighbours from a ring of planes in shared memory, z neighbours
//       carried in registers; mia/3d/image.cc:347-466), the SSD /
//       NCC force (mia/template/ssd.hh:126-181, mia/3d/cost/ncc.cc:88-128),
//       and the transposed spline contraction (translate,
//       spline.cc:731-791): z while walking (four running sums per
//       component, the lowest one final when the window moves on), then x
//       and y in shared memory (the reference contracts y before x; the
//       order changes only the rounding, and x first keeps the intermediate
//       small); the result goes to the tile's partial slot (no atomics).
//   k_gather3         per 4x4x2 block of coefficients: the fixed-order sum of
//       the partial slots that hold each coefficient, the divcurl stencil
//       (C3DPPDivcurlMatrixImpl::evaluate / multiply,
//       mia/3d/ppmatrix.cc:292-599) over a shared-memory copy of the
//       parameters with a 3-node halo, the penalty weight and sign
//       (mia/3d/splinetransformpenalty.cc:60-71) and the full-cost weight
//       (mia/template/fullcost.cxx:37-45).
#include <algorithm>
#include <string>

#include "../../include/mgr.h"
#include "mgr_cost.cuh"
#include "mgr_launch.hh"
#include "warp3_common.cuh"

#include <type_traits>

// the adjoint kernel: resident blocks per SM and planes of its ring (five
// blocks with four planes; six with three, at 72 registers, took 387 instead
// of 382 us per 256^3 NCC evaluation, five planes as long as four)
#ifndef MGR_ADJ_MINB
#define MGR_ADJ_MINB 5
#endif
#define MGR_ADJ_BOUNDS __launch_bounds__(AT3, MGR_ADJ_MINB)
#ifndef MGR_ADJ_PLANES
#define MGR_ADJ_PLANES 4
#endif

namespace mgr {

void set_last_error(const std::string &msg);

namespace {

constexpr int NT3 = 256;   // threads per tile block of the warp kernel: 8 warps
constexpr int AT3 = 128;   // of the adjoint kernel: 4 warps, two rows each
// the adjoint kernel's ring: per warp AD planes of 4 rows of the warped image
// (AD_W floats: x0 - 1 .. x0 + 32, padded) and 2 of the reference
constexpr int AD = MGR_ADJ_PLANES;
constexpr int AD_W = 36;
constexpr int AD_PLANE = 4 * AD_W + 2 * 32;
constexpr int TX3 = 32;    // tile x (lanes)
constexpr int TY3 = 8;     // tile y (warps)
constexpr unsigned FULL = 0xffffffffu;

}  // namespace

// ---------------------------------------------------------------------
// warp
// ---------------------------------------------------------------------
// What bounds it: a sample takes 64 taps from shared memory, a wavefront
// each for the 32 lanes of a warp (about 106 wavefronts per warp step with
// bank conflicts, the tap planes' arrival and the tile's set-up), and the
// instructions around them.  So the walk is kept lean: two planes per step
// whose arithmetic runs on register pairs (one instruction for both), the
// point's integer part from two additions rounded down, a tap address from
// three integer instructions and the ring's wrap from a minimum.  No check
// per voxel: the box that the ring holds contains the taps of every voxel of
// the tile.  192x192x128 SSD, against a walk with scalar arithmetic, a check
// and an index computation per voxel: 435 -> 313 instructions per warp step
// and 77 -> 71 us cold, the shared-memory path 74 -> 81 % busy; evaluations
// one after another 99.3 -> 92.2 us, 256^3 NCC 431 -> 396 us.
//
// COST: the image cost (MGR_COST_SSD / NCC); compiled per cost, the SSD
// kernel keeps one sum and no branch on it.  BATCH: a tile whose box is too
// large for the ring (without the margin below) adds its squares rounded to
// the SSD sum, every other one unrounded: the sums differ in the last bits,
// and a batch's line searches would take other steps
template <int TZ, int COST, bool BATCH>
__device__ __forceinline__ void warp3_body(const EvalArgs &a, int bx, int by, int bz, int tile)
{
    constexpr int NW = NT3 / 32;
    constexpr int NPAIR = RING_N / 2;                      // the ring's slots are filled in pairs of planes
    constexpr unsigned PLANE_B = RING_PLANE * 4u, RING_B = RING_N * PLANE_B;
    static_assert(RING_N % 2 == 0, "pairs of planes");
    constexpr int cost = COST;
    // [RING_N][RING_Y][RING_X] ring (the tensor copies want a 128-byte
    // aligned destination), then C and Tx
    extern __shared__ __align__(128) float sm3[];
    __shared__ float wsum[5][NW];
    __shared__ float csc[2];   // NCC centres (converted once per block)
    __shared__ int zs[TZ];
    __shared__ float4 zw[TZ][2];          // the weights, each twice: {x, x, y, y}, {z, z, w, w}
    __shared__ float urng[6][NW];         // per warp: displacement min / max per component
    __shared__ int boxs[NW][3];           // per warp: the box's xs, ylo, zbase
    __shared__ __align__(8) unsigned long long mbar[NPAIR];
    __shared__ unsigned rdone[NPAIR];     // warps done with the slots' current planes
    __shared__ int nissued;               // pairs of planes whose copies were issued
    __shared__ volatile int ring_failed;  // a wait of this block gave up
    __shared__ int launch_failed;         // one of this launch had, when this block started
    const Axis &X = a.ax[0], &Y = a.ax[1], &Z = a.ax[2];
    const int nx = a.n[0], ny = a.n[1], nz = a.n[2];
    const int x0 = bx * TX3, y0 = by * TY3, z0 = bz * TZ;
    const int ey = min(TY3, ny - y0);
    const int FX = X.fc, FY = Y.fc, FZ = Z.fc;
    const int ncx = a.nc[0], ncy = a.nc[1], ncz = a.nc[2];
    const int tid = threadIdx.x, lane = tid & 31, wy = tid >> 5;
    const int ez = min(TZ, nz - z0);
    // every table entry and scalar the tile needs, loaded up front so that
    // the loads overlap (the data is cold at the start of an evaluation)
    const int cx0 = X.ftile0[bx], cy0 = Y.ftile0[by], cz0 = Z.ftile0[bz];
    const int x = min(x0 + lane, nx - 1), y = min(y0 + wy, ny - 1);
    const int fsx = X.fs[x], fsy = Y.fs[y];
    const float4 fwx = X.fw[x], wyv = Y.fw[y];
    int fsz = 0;
    float4 fwz = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (tid < TZ) {
        const int z = min(z0 + tid, nz - 1);
        fsz = Z.fs[z];
        fwz = Z.fw[z];
    }
    const float mn = a.minmax[0], mxv = a.minmax[1];
    if (tid < 2) csc[tid] = cost == 0 ? 0.0f : float(a.centers[tid]);

    // the parameters' float copy comes from the kernel before this one
    pdl_wait();
    pdl_trigger();
    // whether a wait of this launch has given up (read once: another block may
    // raise the flag meanwhile, and all threads of this one take the same way)
    unsigned flag = 0u;
    if (tid == 0) flag = *(volatile unsigned *)&a.counters[6];
    float *C = sm3 + RING_N * RING_PLANE;  // [3][FZ][FY][FX]
    float *Tx = C + 3 * FZ * FY * FX;      // [3][FZ][FY][32]
    // coefficient footprint: rows (iz, iy) of 3 FX consecutive floats
    // (parameters are interleaved per node), a warp per row, each thread's
    // loads issued as one batch before storing
    for (int j = lane; j < 3 * FX; j += 32) {
        const int ix = j / 3, c = j - 3 * ix;
        const bool inx = cx0 + ix < ncx;
        const float *p = a.params_f + size_t(cx0) * 3 + j;
        float *q = C + c * FZ * FY * FX + ix;
        constexpr int K = 6;
        const int nr = FZ * FY;
        int iz = 0, iy = wy;
        for (int r0 = wy; r0 < nr; r0 += K * NW) {
            float v[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                while (iy >= FY) {
                    iy -= FY;
                    ++iz;
                }
                const bool in = inx && r0 + k * NW < nr && cy0 + iy < ncy && cz0 + iz < ncz;
                v[k] = in ? p[(size_t(cz0 + iz) * ncy + (cy0 + iy)) * ncx * 3] : 0.0f;
                iy += NW;
            }
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (r0 + k * NW < nr) q[(r0 + k * NW) * FX] = v[k];
        }
    }
    if (tid < TZ) {
        zs[tid] = fsz - cz0;
        zw[tid][0] = make_float4(fwz.x, fwz.x, fwz.y, fwz.y);
        zw[tid][1] = make_float4(fwz.z, fwz.z, fwz.w, fwz.w);
    }
    // the ring's barriers: one thread initialises them all (mbarrier and
    // bulk-copy instructions are issued by single threads here)
    if (tid == 0) {
        for (int k = 0; k < NPAIR; ++k) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&mbar[k])) : "memory");
            rdone[k] = 0;
        }
        ring_failed = 0;
        launch_failed = flag != 0u;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    // x stage: Tx[c][kz][jy][lane]
    {
        const int sx = fsx - cx0;
        for (int r = wy; r < 3 * FZ * FY; r += NW) {
            const float *c = C + r * FX + sx;
            Tx[r * 32 + lane] = fwx.x * c[0] + fwx.y * c[1] + fwx.z * c[2] + fwx.w * c[3];
        }
    }
    __syncthreads();
    // y stage on demand: q(c, kz) for this thread's (x, y)
    const int sy = fsy - cy0;
    auto qat = [&](int c, int kz) {
        const float *t = Tx + ((c * FZ + kz) * FY + sy) * 32 + lane;
        return wyv.x * t[0] + wyv.y * t[32] + wyv.z * t[64] + wyv.w * t[96];
    };
    // the window of four z coefficients, components 0 and 1 as pairs
    float2x q01[4];
    float q2[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        q01[m] = pack2(qat(0, m), qat(1, m));
        q2[m] = qat(2, m);
    }
    int cur = 0;   // the window's first z coefficient (zs[0] == 0)
    auto advance = [&](int t) {   // the window moves to the coefficients of plane z0 + t (uniform)
        const int s = zs[t];
        while (cur < s) {
            ++cur;
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                q01[m] = q01[m + 1];
                q2[m] = q2[m + 1];
            }
            q01[3] = pack2(qat(0, cur + 3), qat(1, cur + 3));
            q2[3] = qat(2, cur + 3);
        }
    };
    auto displacement = [&](int t, float &u0, float &u1, float &u2) {
        const float4 wa = zw[t][0], wb = zw[t][1];
        const float2x u01 = fma2(pack2(wb.z, wb.w), q01[3],
                                 fma2(pack2(wb.x, wb.y), q01[2],
                                      fma2(pack2(wa.x, wa.y), q01[0], mul2(pack2(wa.z, wa.w), q01[1]))));
        unpack2(u01, u0, u1);
        u2 = __fmaf_rn(wb.z, q2[3], __fmaf_rn(wb.x, q2[2], __fmaf_rn(wa.x, q2[0], __fmul_rn(wa.z, q2[1]))));
    };
    const bool inxy = (x0 + lane < nx) && (y0 + wy < ny);
    {
        // the range of u over the tile: along z, u is a combination of this
        // thread's q values over the window range 0 .. zs[ez-1] + 3 with
        // non-negative weights summing to 1 (to less than 1 on the last
        // plane of the image, where 0 joins the range).  A NaN stays in the
        // range (the tile is then not staged).
        float lo[3], hi[3];
        float m0[4], m1[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) unpack2(q01[m], m0[m], m1[m]);   // the window's q values are kz = 0..3
        const float *const w4[3] = {m0, m1, q2};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] = min_nan(min_nan(w4[c][0], w4[c][1]), min_nan(w4[c][2], w4[c][3]));
            hi[c] = max_nan(max_nan(w4[c][0], w4[c][1]), max_nan(w4[c][2], w4[c][3]));
        }
        const int kend = zs[ez - 1] + 3;
        for (int kz = 4; kz <= kend; ++kz)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float v = qat(c, kz);
                lo[c] = min_nan(lo[c], v);
                hi[c] = max_nan(hi[c], v);
            }
        const bool last_plane = z0 + ez == nz;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (last_plane) {
                lo[c] = min_nan(lo[c], 0.0f);
                hi[c] = max_nan(hi[c], 0.0f);
            }
            if (!inxy) {
                lo[c] = 3.0e38f;
                hi[c] = -3.0e38f;
            }
            const float l = warp_min_nan(lo[c]), h = warp_max_nan(hi[c]);
            if (lane == 0) {
                urng[c][wy] = l;
                urng[3 + c][wy] = h;
            }
        }
    }
    __syncthreads();
    // tap box of the tile, the same in every thread: x from xs (16-byte
    // aligned in the padded rows), rows from ylo, planes zbase .. zbase +
    // nplanes - 1 of which step t needs t .. t + span - 1
    constexpr int H = PAD_H;
    bool staged, rounded;   // rounded: the squares of planes not walked (BATCH)
    int xs, ylo, zbase, nplanes, span;
    {
        float ulo[3], uhi[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            ulo[c] = warp_min_nan(urng[c][lane & (NW - 1)]);
            uhi[c] = warp_max_nan(urng[3 + c][lane & (NW - 1)]);
        }
        // taps of a voxel at p = v - u: floor(p) - 1 .. floor(p) + 2.  The
        // fixed-point floor may round p up to the next integer: one more
        // row / column / plane on the upper side, which also covers the
        // rounding of u and p there; on the lower side the margin m covers
        // it (u: a few roundings of 2^-24 relative; p: one).
        const float big = 1.0e6f;
        // once a wait of this launch has given up (the flag the host reads
        // afterwards), later blocks read their taps from global memory, so
        // that a stalled copy engine costs one wait limit per launch, not
        // one per block
        bool ok = a.has_tmap != 0 && launch_failed == 0 && (smem_u32(sm3) & 127u) == 0u;
        float m = 0.0f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            ok = ok && fabsf(ulo[c]) < big && fabsf(uhi[c]) < big;
            m = fmaxf(m, fmaxf(fabsf(ulo[c]), fabsf(uhi[c])));
        }
        m = 1.0e-4f + 1.0e-6f * (m + float(max(nx, max(ny, nz))));
        auto fits = [&](float margin) {
            const int xlo = int(floorf(float(x0) - uhi[0] - margin)) - 1;
            const int xe = int(floorf(float(x0 + TX3 - 1) - ulo[0])) + 3;
            xs = ((xlo + H) & ~3) - H;
            ylo = int(floorf(float(y0) - uhi[1] - margin)) - 1;
            const int yhi = int(floorf(float(y0 + ey - 1) - ulo[1])) + 3;
            const int dzl = int(floorf(-uhi[2] - margin)) - 1;
            const int dzh = int(floorf(-ulo[2])) + 3;
            zbase = z0 + dzl;
            span = dzh - dzl + 1;
            nplanes = ez + span - 1;
            return xs >= -H && xe <= nx + H - 1 && xe - xs + 1 <= RING_X && ylo >= -H && yhi <= ny + H - 1 &&
                   yhi - ylo + 1 <= RING_Y && z0 + dzl >= -H && z0 + ez - 1 + dzh <= nz + H - 1 &&
                   span <= RING_N - 2;
        };
        xs = ylo = zbase = nplanes = span = 0;
        staged = ok && fits(m);
        rounded = BATCH && COST == MGR_COST_SSD && !staged && !(ok && fits(0.0f));
    }
    if (lane == 0) {   // for the refills this lane may issue
        boxs[wy][0] = xs + H;
        boxs[wy][1] = ylo + H;
        boxs[wy][2] = zbase + H;
    }
    // one thread: pair k of the box's planes into its ring slots, one tensor
    // copy a plane, completion counted on the pair's mbarrier
    auto issue_pair = [&](int k) {
        const int slot = k % NPAIR;
        const unsigned mb = smem_u32(&mbar[slot]);
        const int np = min(2, nplanes - 2 * k);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(mb), "r"(PLANE_B * unsigned(np))
                     : "memory");
        for (int j = 0; j < np; ++j)
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, "
                "%4}], [%5];\n" ::"r"(smem_u32(sm3) + unsigned(2 * slot + j) * PLANE_B),
                "l"(reinterpret_cast<unsigned long long>(&a.tmap)), "r"(boxs[wy][0]), "r"(boxs[wy][1]),
                "r"(boxs[wy][2] + 2 * k + j), "r"(mb)
                : "memory");
    };
    // the box's first planes, issued by thread 0: the other warps start
    // their walks meanwhile, their waits on a plane end once its copy has
    // been issued and has landed
    if (tid == 0) {
        const int n0 = staged ? min((nplanes + 1) / 2, NPAIR) : 0;
        nissued = n0;
        // (a persistent block's ring was read for the item before)
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        for (int k = 0; k < n0; ++k) issue_pair(k);
    }

    const float px0 = float(x0 + lane), py0 = float(y0 + wy);
    const float ca = csc[0], cb = csc[1];
    const size_t nxy = size_t(nx) * ny;
    const size_t col = size_t(y) * nx + x + size_t(z0) * nxy;
    float acc[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    auto add_cost = [&](float wv, float b, bool round) {
        if (cost == 0) {
            const float d = wv - b;
            acc[0] = round ? __fadd_rn(acc[0], __fmul_rn(d, d)) : __fmaf_rn(d, d, acc[0]);
        } else {
            const float da = wv - ca, db = b - cb;
            acc[0] += da;
            acc[1] += db;
            acc[2] += da * da;
            acc[3] += db * db;
            acc[4] += da * db;
        }
    };
    int tdone = 0;   // planes walked (a warp whose wait gives up stops)
    int kw = 0;      // pairs of planes that have arrived (thread 0 drains from here)
    if (staged) {
        float *wout = a.warped + col;
        const float *rin = a.ref + col;
        // the reference is streamed two steps ahead of its use, so the walk
        // does not wait on its memory latency
        float r0 = 0.0f, r1 = 0.0f, r2 = 0.0f, r3 = 0.0f;
        if (inxy) {
            r0 = __ldg(rin);
            if (ez > 1) r1 = __ldg(rin + nxy);
            if (ez > 2) r2 = __ldg(rin + 2 * nxy);
            if (ez > 3) r3 = __ldg(rin + 3 * nxy);
        }
        // byte offset of a point's first tap in the ring from the bits of its
        // integer parts (floor2): 4 (fx - 1 - xs) + 256 (fy - 1 - ylo) + the
        // plane fz - 1 - zbase; koff also takes off the ring's whole turns
        unsigned koff = 0u - (FLOOR_BITS + 1u + unsigned(xs)) * 4u - (FLOOR_BITS + 1u + unsigned(ylo)) * (RING_X * 4u) -
                        (FLOOR_BITS + 1u + unsigned(zbase)) * PLANE_B;
        // (the last minimum only keeps a wild offset inside the ring)
        auto tap0 = [&](unsigned ix, unsigned iy, unsigned iz) {
            const unsigned o = ix * 4u + iy * (RING_X * 4u) + iz * PLANE_B + koff;
            return min(min(o, o - RING_B), RING_B - 4u);
        };
        auto next_plane = [](unsigned o) { return min(o + PLANE_B, o + PLANE_B - RING_B); };
        unsigned wmb = smem_u32(mbar), wpar = 0;   // the barrier and parity of pair kw
        float zf = float(z0);
        int st = 0;   // the ring slot of plane t
#pragma unroll 1
        for (int t = 0; t < ez; t += 2) {
            const bool two = t + 1 < ez;
            const int tb = two ? t + 1 : t;   // an odd last plane is sampled twice, the second discarded
            float ua0, ua1, ua2, ub0, ub1, ub2;
            advance(t);
            displacement(t, ua0, ua1, ua2);
            advance(tb);
            displacement(tb, ub0, ub1, ub2);
            const int need = min((t + span) >> 1, (nplanes - 1) >> 1);
            bool failed = false;
            while (kw <= need) {
                if (!mbar_wait(wmb, wpar) || ring_failed) {
                    failed = true;
                    break;
                }
                ++kw;
                wmb += 8;
                if (wmb == smem_u32(mbar) + 8 * NPAIR) {
                    wmb = smem_u32(mbar);
                    wpar ^= 1u;
                }
            }
            if (failed) {
                if (!ring_failed) {
                    ring_failed = 1;
                    atomicOr(&a.counters[6], 1u);
                }
                // lanes of this warp whose waits did not give up walk on, and
                // wait for this one wherever they release planes
                for (; t < ez && t + RING_N < nplanes; t += 2) __syncwarp();
                break;
            }
            const float2x px = pack2(px0 - ua0, px0 - ub0), py = pack2(py0 - ua1, py0 - ub1);
            const float2x pz = pack2(zf - ua2, (two ? zf + 1.0f : zf) - ub2);
            unsigned xa, xb, ya, yb, za, zb;
            const float2x fx = floor2(px, xa, xb), fy = floor2(py, ya, yb), fz = floor2(pz, za, zb);
            unsigned oa = tap0(xa, ya, za), ob = tap0(xb, yb, zb);
            float2x wx[4], wyp[4], wz[4];
            bspline3_weights2(sub2(px, fx), wx);
            bspline3_weights2(sub2(py, fy), wyp);
            bspline3_weights2(sub2(pz, fz), wz);
            float2x sum;
#pragma unroll
            for (int kz = 0; kz < 4; ++kz) {
                const float *pa = reinterpret_cast<const float *>(reinterpret_cast<const char *>(sm3) + oa);
                const float *pb = reinterpret_cast<const float *>(reinterpret_cast<const char *>(sm3) + ob);
                float2x ay;
#pragma unroll
                for (int ky = 0; ky < 4; ++ky) {
                    const float *ra = pa + ky * RING_X, *rb = pb + ky * RING_X;
                    float2x r = mul2(wx[1], pack2(ra[1], rb[1]));
                    r = fma2(wx[0], pack2(ra[0], rb[0]), r);
                    r = fma2(wx[2], pack2(ra[2], rb[2]), r);
                    r = fma2(wx[3], pack2(ra[3], rb[3]), r);
                    ay = ky == 0 ? mul2(wyp[0], r) : fma2(wyp[ky], r, ay);
                }
                sum = kz == 0 ? mul2(wz[0], ay) : fma2(wz[kz], ay, sum);
                oa = next_plane(oa);
                ob = next_plane(ob);
            }
            if (inxy) {
                float wa, wb;
                unpack2(sum, wa, wb);
                wa = fminf(fmaxf(wa, mn), mxv);
                wb = fminf(fmaxf(wb, mn), mxv);
                wout[0] = wa;
                add_cost(wa, r0, false);
                if (two) {
                    wout[nxy] = wb;
                    add_cost(wb, r1, false);
                }
            }
            r0 = r2;
            r1 = r3;
            if (inxy && t + 4 < ez) r2 = __ldg(rin + 4 * nxy);
            if (inxy && t + 5 < ez) r3 = __ldg(rin + 5 * nxy);
            wout += 2 * nxy;
            rin += 2 * nxy;
            zf += 2.0f;
            tdone = tb + 1;
            // this warp is done with planes t and t + 1; the last warp
            // refills their slots
            if (t + RING_N < nplanes) {
                __syncwarp();
                if (lane == 0) {
                    __threadfence_block();
                    if (atomicAdd(&rdone[st >> 1], 1u) == unsigned(NW - 1)) {
                        rdone[st >> 1] = 0;
                        if (!ring_failed) {
                            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                            issue_pair((t + RING_N) >> 1);
                            atomicAdd(&nissued, 1);
                        }
                    }
                }
            }
            st += 2;
            if (st == RING_N) {
                st = 0;
                koff -= RING_B;
            }
        }
    }
    // the planes not walked (a tile whose taps do not fit the ring, or the
    // rest of a walk whose wait gave up): the displacement from the y stage's
    // window at plane t (the walk's values: the window then starts at
    // coefficient zs[t]) and the taps from global memory.  They come after
    // the walk, so that the walk itself makes no call (a call site costs the
    // loop register spills).
    if (inxy)
        for (int t = tdone; t < ez; ++t) {
            const int s = zs[t];
            const float4 wa = zw[t][0], wb = zw[t][1];
            float u[3];
#pragma unroll
            for (int c = 0; c < 3; ++c)
                u[c] = wa.x * qat(c, s) + wa.z * qat(c, s + 1) + wb.x * qat(c, s + 2) + wb.z * qat(c, s + 3);
            const float wv = taps3_global(a, px0 - u[0], py0 - u[1], float(z0 + t) - u[2], mn, mxv);
            a.warped[col + size_t(t) * nxy] = wv;
            add_cost(wv, __ldg(a.ref + col + size_t(t) * nxy), rounded);
        }
    // tile sums: a float tree within each warp (5 levels), the warps' sums
    // added in double in a fixed order, one thread per sum (FP64 is slow
    // here, so it is kept off the per-thread path)
    const int ncomp = cost == 0 ? 1 : 5;
#pragma unroll
    for (int k = 0; k < 5; ++k)
        if (k < ncomp) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(FULL, acc[k], o);
            if (lane == 0) wsum[k][wy] = acc[k];
        }
    __syncthreads();   // also: every warp is done with the ring
    if (staged && tid == 0) {
        // copies still in flight (only after a wait gave up) are waited for
        // before the block's shared memory is released: only the planes that
        // were issued, and within one wait limit in total (a pair whose
        // wait gives up ends the drain)
        const int issued = nissued;
        for (; kw < issued; ++kw)
            if (!mbar_wait(smem_u32(&mbar[kw % NPAIR]), unsigned(kw / NPAIR) & 1u)) {
                atomicOr(&a.counters[6], 1u);
                break;
            }
    }
    // a persistent block's next item initialises the barriers again, for which
    // they have to be invalidated first
    if (BATCH && tid == 0)
        for (int k = 0; k < NPAIR; ++k)
            asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_u32(&mbar[k])) : "memory");
    if (tid < 5) {
        double v = 0.0;
        if (tid < ncomp)
            for (int w = 0; w < NW; ++w) v += widen(wsum[tid][w]);
        a.tile_sums[size_t(tile) * 5 + tid] = v;
    }
    // (the cost is finalised from the tile sums after this kernel: an SSD cost
    // by the gather, an NCC cost by k_finalise3; a last-block pass here, even
    // one that is not taken, cost 383x351x317 SSD 662 instead of 654 us)
}

// ---------------------------------------------------------------------
// gradient + force + adjoint
// ---------------------------------------------------------------------
// A thread walks two columns, rows 2w and 2w + 1 of the tile for warp w: the
// two rows' arithmetic runs on register pairs, they share the loop, the
// tables and each other's values.  Each warp copies the planes it needs (its
// rows, the ones above and below, the rows' ends, the reference) into a ring
// of its own, ahead of the walk and without a block barrier.  What bounds the
// walk is the latency of those reads, one plane after another: with loads a
// plane ahead in registers a plane took 0.7 us.  Where the image ends, a
// neighbour's offset names the voxel that makes the difference 0 (y), or a
// second scale is 0 (x), so the walk has no branch on it.  Against one row per
// thread with loads at their use, alone on the GPU: 256^3 NCC 93 -> 74 us,
// 383x351x317 SSD 180 -> 137 us; 192x192x128 SSD 30 -> 29 us (1008 tiles are
// 1.3 waves, a block's chain of stages is its time).
template <int TZ>
__device__ __forceinline__ void adjoint3_body(const EvalArgs &a, int bx, int by, int bz, int tile_index)
{
    const int cost = a.cost;
    extern __shared__ __align__(16) float sm3a[];
    __shared__ int asx[TX3], asy[TY3], azs[TZ];
    __shared__ float fsc[5];   // force constants (converted once per block)
    __shared__ float4 awx[TX3][2], awy[TY3][2], azw[TZ][2];   // each weight twice, {x, x, y, y}, {z, z, w, w}
    const Axis &X = a.ax[0], &Y = a.ax[1], &Z = a.ax[2];
    const int nx = a.n[0], ny = a.n[1], nz = a.n[2];
    const int x0 = bx * TX3, y0 = by * TY3, z0 = bz * TZ;
    const int ey = min(TY3, ny - y0), ez = min(TZ, nz - z0);
    const int AXc = X.ac, AYc = Y.ac, AZc = Z.ac;
    const int ax0 = X.atile0[bx], ay0 = Y.atile0[by], az0 = Z.atile0[bz];
    const int tid = threadIdx.x, lane = tid & 31, wy = tid >> 5;
    float *part = a.partial + size_t(tile_index) * a.slot;
    constexpr int AZP = TX3 + 1;              // Az row pitch (odd: the x stage reads along the rows)
    float2x *Az = reinterpret_cast<float2x *>(sm3a);                   // [3][AZc][4][AZP], the rows in pairs
    float *Ax = sm3a + 3 * AZc * TY3 * AZP;                            // [3][AZc][8][AXc], in the ring's place
    float *ring = sm3a + 3 * AZc * TY3 * AZP + wy * (AD * AD_PLANE);   // [AD][AD_PLANE] of this warp

    // tables and scalars, loaded up front
    auto twice = [](float4 (&d)[2], const float4 &w) {
        d[0] = make_float4(w.x, w.x, w.y, w.y);
        d[1] = make_float4(w.z, w.z, w.w, w.w);
    };
    if (tid < TX3) {
        const int xx = min(x0 + tid, nx - 1);
        asx[tid] = X.as[xx] - ax0;
        twice(awx[tid], X.aw[xx]);
    } else if (tid < TX3 + TY3) {
        const int k = tid - TX3, yy = min(y0 + k, ny - 1);
        asy[k] = Y.as[yy] - ay0;
        twice(awy[k], Y.aw[yy]);
    } else if (tid >= 64 && tid < 64 + TZ) {
        const int k = tid - 64, zz = min(z0 + k, nz - 1);
        azs[k] = Z.as[zz] - az0;
        twice(azw[k], Z.aw[zz]);
    }
    // the two columns (clamped to the image; their scale is 0 beyond it) and
    // the offsets of their neighbours in a plane
    const int x = x0 + lane, ya = y0 + 2 * wy, yb = ya + 1;
    const size_t nxy = size_t(nx) * ny;
    const int xc = min(x, nx - 1);
    const unsigned oa = unsigned(min(ya, ny - 1) * nx + xc), ob = unsigned(min(yb, ny - 1) * nx + xc);
    const unsigned ou = ya > 0 && ya < ny - 1 ? oa - unsigned(nx) : ob;   // above row a (row b is below it)
    const unsigned od = yb < ny - 1 ? ob + unsigned(nx) : oa;             // below row b (row a is above it)
    // lanes 0..3 also copy the rows' ends: (row a, row b) x (left, right)
    const int xe = lane & 1 ? min(x0 + TX3, nx - 1) : max(x0 - 1, 0);
    const unsigned oe = (lane & 2 ? ob : oa) - unsigned(xc) + unsigned(xe);
    const float *wsrc = a.warped + size_t(z0) * nxy;   // the next plane to copy
    const float *rsrc = a.ref + size_t(z0) * nxy;
    const unsigned sring = smem_u32(ring) + 4u * unsigned(lane);
    const unsigned sedge = smem_u32(ring) + 4u * unsigned((lane & 2 ? 2 : 1) * AD_W + (lane & 1 ? TX3 + 1 : 0));
    // (lanes beyond the image get zeros: many lanes copying from one address
    // take turns, 130x120x110 SSD 61.4 instead of 52.4 us an evaluation)
    const int bytes = x < nx ? 4 : 0;
    auto copy4 = [](unsigned dst, const float *src, int n) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
    };
    // plane p of the tile into its slot: those the walk reads, up to the one
    // behind the last if the image has it; a group is committed for every p
    const int np = min(ez + 1, nz - z0);
    auto issue = [&](int p, unsigned slot) {
        if (p < np) {
            const unsigned d = sring + slot;
            copy4(d + 4u, wsrc + ou, bytes);
            copy4(d + 4u * (AD_W + 1), wsrc + oa, bytes);
            copy4(d + 4u * (2 * AD_W + 1), wsrc + ob, bytes);
            copy4(d + 4u * (3 * AD_W + 1), wsrc + od, bytes);
            if (lane < 4) copy4(sedge + slot, wsrc + oe, 4);
            copy4(d + 4u * (4 * AD_W), rsrc + oa, bytes);
            copy4(d + 4u * (4 * AD_W + 32), rsrc + ob, bytes);
            wsrc += nxy;
            rsrc += nxy;
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // the warped image and the cost's scalars come from the warp kernel
    pdl_wait();
    pdl_trigger();
    float2x wm = 0;
    if (z0 > 0) wm = pack2(__ldcg(wsrc - nxy + oa), __ldcg(wsrc - nxy + ob));
#pragma unroll
    for (int p = 0; p < AD - 1; ++p) issue(p, unsigned(p) * (AD_PLANE * 4u));
    if (tid < 5) {
        // the SSD force scale from the settings, as the finalisation sets it
        // (with a deferred finalisation it is not set yet)
        if (cost != 0) fsc[tid] = float(a.scalars[SC_K1 + tid]);
        else if (tid == 4) fsc[4] = a.ssd_norm ? float(1.0 / double(size_t(nx) * ny * nz)) : 1.0f;
    }
    asm volatile("cp.async.wait_group %0;\n" ::"n"(AD - 2) : "memory");   // plane 0
    __syncthreads();
    // central differences are taken without their factor 1/2, which joins
    // the force's scale
    const bool ina = x < nx && ya < ny, inb = x < nx && yb < ny;
    float2x hs, k1 = 0, k2 = 0, ma = 0, mb = 0;
    if (cost == 0) {
        const float h = 0.5f * fsc[4];
        hs = pack2(ina ? h : 0.0f, inb ? h : 0.0f);
    } else {
        hs = pack2(ina ? 0.5f : 0.0f, inb ? 0.5f : 0.0f);
        k1 = pack2(fsc[0], fsc[0]);
        k2 = pack2(fsc[1], fsc[1]);
        ma = pack2(fsc[2], fsc[2]);
        mb = pack2(fsc[3], fsc[3]);
    }

    const float2x hx = x > 0 && x < nx - 1 ? hs : 0;   // no x difference at the image's border

    float2x acc[3][4];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[c][k] = 0;
    int cur = 0;   // azs[0] == 0
    float2x *const az = Az + wy * AZP + lane;
    auto emit = [&](int kz, int c, float2x v) { az[(c * AZc + kz) * (TY3 / 2 * AZP)] = v; };
    const float *rp = ring + lane;   // plane t's slot
    float2x w0 = pack2(rp[AD_W + 1], rp[2 * AD_W + 1]);
    unsigned fill = (AD - 1) * (AD_PLANE * 4u);   // the slot that plane t - 1 has left
    int at = 0;                                   // t modulo AD
#pragma unroll 1
    for (int t = 0; t < ez; ++t) {
        const int z = z0 + t;
        issue(t + AD - 1, fill);
        fill = fill == (AD - 1) * (AD_PLANE * 4u) ? 0u : fill + AD_PLANE * 4u;
        asm volatile("cp.async.wait_group %0;\n" ::"n"(AD - 2) : "memory");   // plane t + 1
        __syncwarp();
        at = at == AD - 1 ? 0 : at + 1;
        const float *rn = ring + at * AD_PLANE + lane;
        const float2x wp = pack2(rn[AD_W + 1], rn[2 * AD_W + 1]);
        const float2x left = pack2(rp[AD_W], rp[2 * AD_W]), right = pack2(rp[AD_W + 2], rp[2 * AD_W + 2]);
        const float up = rp[1], down = rp[3 * AD_W + 1];
        const float2x b = pack2(rp[4 * AD_W], rp[4 * AD_W + 32]);
        rp = rn;
        __syncwarp();   // every lane has plane t: its slot is free
        float wa, wb;
        unpack2(w0, wa, wb);
        // the force's factor at the voxel, times the scale
        float2x d;
        if (cost == 0)
            d = sub2(w0, b);
        else
            d = mul2(k1, fma2(k2, sub2(w0, ma), sub2(mb, b)));
        const float2x s = mul2(d, hs);
        float2x f[3];
        f[0] = mul2(sub2(right, left), mul2(d, hx));
        f[1] = mul2(sub2(pack2(wb, down), pack2(up, wa)), s);
        f[2] = z > 0 && z < nz - 1 ? mul2(sub2(wp, wm), s) : 0;
        const int sz = azs[t];
        while (cur < sz) {   // uniform over the block
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                emit(cur, c, acc[c][0]);
                acc[c][0] = acc[c][1];
                acc[c][1] = acc[c][2];
                acc[c][2] = acc[c][3];
                acc[c][3] = 0;
            }
            ++cur;
        }
        const float4 u = azw[t][0], v = azw[t][1];
        const float2x w4[4] = {pack2(u.x, u.y), pack2(u.z, u.w), pack2(v.x, v.y), pack2(v.z, v.w)};
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[c][k] = fma2(w4[k], f[c], acc[c][k]);
        wm = w0;
        w0 = wp;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (cur + k < AZc)
#pragma unroll
            for (int c = 0; c < 3; ++c) emit(cur + k, c, acc[c][k]);
    for (int kz = cur + 4; kz < AZc; ++kz)
#pragma unroll
        for (int c = 0; c < 3; ++c) emit(kz, c, 0);
    __syncthreads();
    // the transposed contraction of a line of `len` pairs onto nout
    // coefficients as a sliding window of four sums (the starts are the same
    // for every thread, so the window moves in lock step); entry l of the
    // line from in(l), coefficient o to out(o, sum)
    auto contract = [](int len, const int *start, const float4 (*w)[2], int nout, auto in, auto out) {
        float2x s0 = 0, s1 = 0, s2 = 0, s3 = 0;
        int oc = 0;
        auto step = [&](int l) {
            const int o = start[l];
            while (oc < o) {
                out(oc, s0);
                s0 = s1;
                s1 = s2;
                s2 = s3;
                s3 = 0;
                ++oc;
            }
            const float4 u = w[l][0], v = w[l][1];
            const float2x f = in(l);
            s0 = fma2(pack2(u.x, u.y), f, s0);
            s1 = fma2(pack2(u.z, u.w), f, s1);
            s2 = fma2(pack2(v.x, v.y), f, s2);
            s3 = fma2(pack2(v.z, v.w), f, s3);
        };
        int l = 0;
        for (; l + 8 <= len; l += 8)
#pragma unroll
            for (int j = 0; j < 8; ++j) step(l + j);
        for (; l < len; ++l) step(l);
        if (oc < nout) out(oc, s0);
        if (oc + 1 < nout) out(oc + 1, s1);
        if (oc + 2 < nout) out(oc + 2, s2);
        if (oc + 3 < nout) out(oc + 3, s3);
        for (int o = oc + 4; o < nout; ++o) out(o, 0);
    };
    // x stage, one thread per (c, kz, row pair) line of Az, all TX3 columns
    // (the walk leaves 0 in the columns beyond the image, whose coefficient
    // start is the last column's).  Contracting x before y keeps the
    // intermediate small (AXc instead of 32 values per row): the block needs
    // less shared memory and the two stages fewer instructions.
    for (int e = tid; e < 3 * AZc * (TY3 / 2); e += AT3) {
        if (2 * (e & (TY3 / 2 - 1)) >= ey) continue;   // rows below the image: never read
        const float2x *src = Az + e * AZP;
        float *dst = Ax + 2 * e * AXc;
        contract(TX3, asx, awx, AXc, [&](int l) { return src[l]; },
                 [&](int o, float2x v) { unpack2(v, dst[o], dst[AXc + o]); });
    }
    __syncthreads();
    // y stage, one thread per two (c, kz, ix) columns of Ax, straight into the
    // partial slot ((kz AYc + jy) AXc + ix) 3 + c
    const int ncol = 3 * AZc * AXc, half = (ncol + 1) / 2;
    auto column = [&](int q, const float *&src, float *&dst) {
        const int r = q / AXc, ix = q - r * AXc;   // r = c AZc + kz
        const int c = r / AZc, kz = r - c * AZc;
        src = Ax + r * TY3 * AXc + ix;
        dst = part + (size_t(kz) * AYc * AXc + ix) * 3 + c;
    };
    for (int e = tid; e < half; e += AT3) {
        const bool two = e + half < ncol;
        const float *src0, *src1;
        float *dst0, *dst1;
        column(e, src0, dst0);
        column(two ? e + half : e, src1, dst1);
        contract(ey, asy, awy, AYc, [&](int l) { return pack2(src0[l * AXc], src1[l * AXc]); },
                 [&](int o, float2x v) {
                     float p, q;
                     unpack2(v, p, q);
                     dst0[o * AXc * 3] = p;
                     if (two) dst1[o * AXc * 3] = q;
                 });
    }
}

// ---------------------------------------------------------------------
// gather + penalty
// ---------------------------------------------------------------------
#ifndef MGR_GATHER_THREADS
#define MGR_GATHER_THREADS 256
#endif
#ifndef MGR_GATHER_MINB
#define MGR_GATHER_MINB 4
#endif
#define MGR_GATHER_BOUNDS __launch_bounds__(MGR_GATHER_THREADS, MGR_GATHER_MINB)
namespace {
constexpr int GT3 = MGR_GATHER_THREADS;
constexpr int GBX = 4, GBY = 4, GBZ = 2;   // coefficients per block: 32, lane = coefficient
constexpr int GH = 3;                      // stencil half width
constexpr int GPX = GBX + 2 * GH;          // 10: halo tile edges
constexpr int GPY = GBY + 2 * GH;          // 10
constexpr int GPZ = GBZ + 2 * GH;          // 8
constexpr int GPP = 12;                    // padded row pitch (float4) of the halo tile
constexpr int GSUB = GT3 / 32;             // the warps split each coefficient's work
constexpr int GNQ = 12;                    // per-warp partials: 9 penalty products, 3 image sums
constexpr int GSMAX = 64 / GSUB;           // partial slots per warp loaded in the first batch
// the per-warp partials fit beside the halo tables at 8 warps; with more
// warps they take the tables' place once the stencil is summed
constexpr int GTAB = GPZ * GPY * GPP + 343 * 2;   // float4: Ps, then Pt
constexpr bool GALIAS = GSUB * GNQ * 32 > 12 * 32 * 8;
static_assert(!GALIAS || GSUB * GNQ * 32 <= 4 * GTAB, "partials must fit in the tables' space");
}  // namespace

// Block: 4 x 4 x 2 coefficients, one per lane; the 8 warps split the 49
// (dz, dy) rows of the 7^3 divcurl stencil and the partial slots.  Loads are
// issued in two batches: the tables, the parameters with a 3-node halo and
// the penalty cells; then the partial slots, in flight while the stencil
// is summed.
// A block's chain of steps is the kernel's time on small grids, so its end is
// short: a warp per gradient component, one for the value, whose thread
// arrives with no other store in flight, no FP64 but the sums, and a last
// block whose loads are in flight together.  40x44x36 NCC, alone on the GPU:
// 13.1 -> 11.7 us (of 29.8 k cycles 10 k were the end, 6 k the last block);
// evaluations one after another 13.8 -> 13.0 us, the value alone of
// 160x176x144 120 -> 117 us.
__device__ __forceinline__ void gather3_body(const EvalArgs &a, int with_gradient, int image_from_dense, int blk,
                                             int nblk)
{
    __shared__ float4 PsPt[GTAB];
    __shared__ float pacc_own[GALIAS ? 1 : GSUB * GNQ * 32];
    __shared__ int gl[3][GBX][GATHER_LMAX];
    __shared__ int gn[3][GBX];
    __shared__ bool is_last;
    float4 *Ps = PsPt, *Pt = PsPt + GPZ * GPY * GPP;
    float (*pacc)[GNQ][32] = reinterpret_cast<float (*)[GNQ][32]>(GALIAS ? reinterpret_cast<float *>(PsPt) : pacc_own);
    const Axis &X = a.ax[0], &Y = a.ax[1], &Z = a.ax[2];
    const int ncx = a.nc[0], ncy = a.nc[1], ncz = a.nc[2];
    const int nbx = (ncx + GBX - 1) / GBX, nby = (ncy + GBY - 1) / GBY;
    const int bxi = blk % nbx, byi = (blk / nbx) % nby, bzi = blk / (nbx * nby);
    const int cx0 = bxi * GBX, cy0 = byi * GBY, cz0 = bzi * GBZ;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int lx = lane & 3, ly = (lane >> 2) & 3, lz = lane >> 4;
    const int cx = cx0 + lx, cy = cy0 + ly, cz = cz0 + lz;
    const bool valid = cx < ncx && cy < ncy && cz < ncz;
    const size_t i = valid ? (size_t(cz) * ncy + cy) * ncx + cx : 0;
    const bool img = with_gradient && !image_from_dense;

    // fixed tables first: offset lists and penalty cells
    if (img) {
        if (tid < 3 * GBX) {
            const int ax = tid / GBX, k = tid - ax * GBX;
            const int c = (ax == 0 ? cx0 : ax == 1 ? cy0 : cz0) + k;
            gn[ax][k] = c < a.nc[ax] && (ax < 2 || k < GBZ) ? a.ax[ax].glen[c] : 0;
        }
        // whole lists (0 past their length), every entry by a thread of its own
        for (int e = tid; e < 3 * GBX * GATHER_LMAX; e += GT3) {
            const int ax = e / (GBX * GATHER_LMAX), r = e - ax * (GBX * GATHER_LMAX), k = r / GATHER_LMAX;
            const int base = ax == 0 ? cx0 : ax == 1 ? cy0 : cz0;
            if (base + k < a.nc[ax]) gl[ax][k][r - k * GATHER_LMAX] = a.ax[ax].glist[size_t(base) * GATHER_LMAX + r];
        }
    }
    if (a.has_penalty) {
        constexpr int KT = (343 + GT3 - 1) / GT3;
        float tv[KT][6];
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            const int e = tid + k * GT3;
            if (e < 343) {
                const int dx = e % 7 - 3, dy = (e / 7) % 7 - 3, dz = e / 49 - 3;
                const float *P = a.ptable + (((dz + 4) * 9 + (dy + 4)) * 9 + (dx + 4)) * 6;
#pragma unroll
                for (int j = 0; j < 6; ++j) tv[k][j] = P[j];
            }
        }
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            const int e = tid + k * GT3;
            if (e < 343) {
                Pt[2 * e] = make_float4(tv[k][0], tv[k][1], tv[k][2], tv[k][3]);
                Pt[2 * e + 1] = make_float4(tv[k][4], tv[k][5], 0.0f, 0.0f);
            }
        }
    }
    // The divcurl stencil needs only the parameters' float copy, which
    // every launch order of this kernel has completed before any block of
    // it starts (the conversion kernel is never launched directly before
    // it; the kernel between them waits for the conversion before it lets
    // this one launch).  So the stencil runs before the dependency wait,
    // while the adjoint kernel finishes; the copy is read through the L2
    // (ld.global.cg), never from a line an earlier kernel left in L1.
    if (a.has_penalty) {
        constexpr int NH = GPX * GPY * GPZ;
        constexpr int KP = (NH + GT3 - 1) / GT3;
        float pv[KP][3];
#pragma unroll
        for (int k = 0; k < KP; ++k) {
            const int e = tid + k * GT3;
            pv[k][0] = pv[k][1] = pv[k][2] = 0.0f;
            if (e < NH) {
                const int hx = e % GPX, hy = (e / GPX) % GPY, hz = e / (GPX * GPY);
                const int gx = cx0 - GH + hx, gy = cy0 - GH + hy, gz = cz0 - GH + hz;
                if (gx >= 0 && gx < ncx && gy >= 0 && gy < ncy && gz >= 0 && gz < ncz) {
                    const float *p = a.params_f + ((size_t(gz) * ncy + gy) * ncx + gx) * 3;
                    pv[k][0] = __ldcg(p);
                    pv[k][1] = __ldcg(p + 1);
                    pv[k][2] = __ldcg(p + 2);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < KP; ++k) {
            const int e = tid + k * GT3;
            if (e < NH) {
                const int hx = e % GPX, hy = (e / GPX) % GPY, hz = e / (GPX * GPY);
                Ps[(hz * GPY + hy) * GPP + hx] = make_float4(pv[k][0], pv[k][1], pv[k][2], 0.0f);
            }
        }
    }
    __syncthreads();   // the offset lists, the parameter halo
    // R0..R5, T0..T2: the nine products of the 3x3 cell with c_j, summed
    // over the 7^3 neighbours j = i - d (zero outside the grid)
    float R0 = 0, R1 = 0, R2 = 0, R3 = 0, R4 = 0, R5 = 0, T0 = 0, T1 = 0, T2 = 0;
    if (valid && a.has_penalty) {
        for (int p = w; p < 49; p += GSUB) {
            const int dz = p / 7 - 3, dy = p % 7 - 3;
            const float4 *prow = Ps + ((lz + GH - dz) * GPY + (ly + GH - dy)) * GPP + (lx + GH);
            const float4 *trow = Pt + p * 14;
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                const float4 cj = prow[3 - k];     // dx = k - 3
                const float4 t0 = trow[2 * k], t1 = trow[2 * k + 1];
                R0 += t0.x * cj.x;
                R1 += t0.y * cj.y;
                R2 += t0.z * cj.y;
                R3 += t0.w * cj.z;
                R4 += t1.x * cj.z;
                R5 += t1.y * cj.x;
                T0 += t1.y * cj.z;
                T1 += t0.y * cj.x;
                T2 += t0.w * cj.y;
            }
        }
    }
    pdl_wait();
    pdl_trigger();
    // parameters the conversion found non-finite: nothing is written to the
    // caller's buffers (read by every block before its arrival)
    const bool bad = a.params_host && *(volatile unsigned *)&a.counters[7] != 0u;
    // the adjoint's partial slots: this warp's share (entries k = w,
    // w + GSUB, ...) of the lane's coefficient, in batches of loads
    constexpr int SMAX = GSMAX;
    int tot = 0, nX = 0, nY = 0, nZ = 0;
    bool lists = false;
    if (valid && img) {
        nX = gn[0][lx];
        nY = gn[1][ly];
        nZ = gn[2][lz];
        lists = nX >= 0 && nY >= 0 && nZ >= 0;
        if (lists) tot = nX * nY * nZ;
    }
    float S0 = 0.0f, S1 = 0.0f, S2 = 0.0f;
    for (int k0 = w; k0 < tot; k0 += GSUB * SMAX) {
        float sv[SMAX][3];
#pragma unroll
        for (int u = 0; u < SMAX; ++u) {
            const int k = k0 + GSUB * u;
            sv[u][0] = sv[u][1] = sv[u][2] = 0.0f;
            if (k < tot) {
                const int jx = k % nX, r = k / nX;
                const int jy = r % nY, jz = r / nY;
                const float *p = a.partial + (size_t(gl[2][lz][jz] + gl[1][ly][jy]) + gl[0][lx][jx]);
                sv[u][0] = p[0];
                sv[u][1] = p[1];
                sv[u][2] = p[2];
            }
        }
#pragma unroll
        for (int u = 0; u < SMAX; ++u) {
            S0 += sv[u][0];
            S1 += sv[u][1];
            S2 += sv[u][2];
        }
    }
    if (valid && img && !lists) {
        const int2 gx = X.gtile[cx], gy = Y.gtile[cy], gz = Z.gtile[cz];
        const int mX = gx.y - gx.x + 1, mY = gy.y - gy.x + 1, mZ = gz.y - gz.x + 1;
        const int mt = (mX > 0 && mY > 0 && mZ > 0) ? mX * mY * mZ : 0;
        for (int k = w; k < mt; k += GSUB) {
            const int tx = gx.x + k % mX, ty = gy.x + (k / mX) % mY, tz = gz.x + k / (mX * mY);
            const int lxo = cx - X.atile0[tx], lyo = cy - Y.atile0[ty], lzo = cz - Z.atile0[tz];
            const size_t t = (size_t(tz) * Y.nt + ty) * X.nt + tx;
            const float *p = a.partial + t * a.slot + ((size_t(lzo) * Y.ac + lyo) * X.ac + lxo) * 3;
            S0 += p[0];
            S1 += p[1];
            S2 += p[2];
        }
    }
    // the lane's own parameters (the penalty value), read before the
    // partials may take the tables' place
    float ci[3] = {0.0f, 0.0f, 0.0f};
    if (w == 3 && a.has_penalty) {
        const float4 c4 = Ps[((lz + GH) * GPY + (ly + GH)) * GPP + (lx + GH)];
        ci[0] = c4.x;
        ci[1] = c4.y;
        ci[2] = c4.z;
    }
    if (GALIAS) __syncthreads();
    pacc[w][0][lane] = R0;
    pacc[w][1][lane] = R1;
    pacc[w][2][lane] = R2;
    pacc[w][3][lane] = R3;
    pacc[w][4][lane] = R4;
    pacc[w][5][lane] = R5;
    pacc[w][6][lane] = T0;
    pacc[w][7][lane] = T1;
    pacc[w][8][lane] = T2;
    pacc[w][9][lane] = S0;
    pacc[w][10][lane] = S1;
    pacc[w][11][lane] = S2;
    __syncthreads();
    // the warps' partials of each quantity summed in a fixed order (FP32,
    // warp k % GSUB sums quantity k into row 0), which the warps below combine
    // (the outputs are widened to double at the store)
    for (int k = w; k < GNQ; k += GSUB) {
        float t = pacc[0][k][lane];
#pragma unroll
        for (int ww = 1; ww < GSUB; ++ww) t += pacc[ww][k][lane];
        pacc[0][k][lane] = t;
    }
    __syncthreads();
    // a warp per component of the gradient, one for the penalty's value and
    // the block's arrival
    __shared__ __align__(16) double gst[32 * 3];
    if (w < 3) {
        if (valid && with_gradient && !bad) {
            const size_t o = i * 3 + w;
            const float gp = a.has_penalty ? a.pen_grad_wf * (pacc[0][6 + w][lane] +
                                                   (2.0f * pacc[0][2 * w][lane] + pacc[0][2 * w + 1][lane]))
                                           : 0.0f;
            const double gi = image_from_dense ? a.grad_image[o] : widen(a.cost_wf * -pacc[0][9 + w][lane]);
            const double gpd = widen(gp), gt = gi + gpd;
            if (a.params_host) gst[lane * 3 + w] = gt;
            else a.grad_total[o] = gt;
            if (a.grad_image && !image_from_dense) a.grad_image[o] = gi;
            if (a.grad_penalty) a.grad_penalty[o] = gpd;
        }
    } else if (w == 3) {
        float pval = 0.0f;
        if (valid && a.has_penalty) {
            float v[7];
#pragma unroll
            for (int k = 0; k < 7; ++k) v[k] = pacc[0][k][lane];
            if (with_gradient)
                pval = ci[0] * v[0] + ci[0] * v[1] + ci[1] * v[2] + ci[1] * v[3] + ci[2] * v[4] + ci[2] * v[5];
            else
                pval = ci[0] * v[0] + ci[1] * v[2] + ci[2] * v[4] + ci[0] * v[1] + ci[0] * v[6] + ci[1] * v[3];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) pval += __shfl_xor_sync(FULL, pval, o);
        if (lane == 0) {
            a.pen_part[blk] = widen(pval);
            is_last = arrive_last(&a.counters[1], nblk);
        }
    }
    __syncthreads();
    if (w == 0 && with_gradient && !bad && a.params_host) {
        // the total gradient into the caller's host memory: the lanes of
        // a row (ly, lz) hold four consecutive coefficients, 96
        // contiguous bytes of the output; a row whose four coefficients
        // are all in the grid and whose start is 16-byte aligned is
        // stored as six 16-byte pieces (few large writes over the
        // CPU-GPU link: an evaluation from host buffers took 153.9
        // instead of 158.0 us at 192x192x128), any other lane stores
        // its own three values
        auto row_dst = [&](int r) -> double * {
            const int ry = cy0 + (r & 3), rz = cz0 + (r >> 2);
            return a.grad_total + ((size_t(rz) * ncy + ry) * ncx + cx0) * 3;
        };
        auto row_vec = [&](int r) -> bool {
            const int ry = cy0 + (r & 3), rz = cz0 + (r >> 2);
            return cx0 + GBX <= ncx && ry < ncy && rz < ncz && (reinterpret_cast<uintptr_t>(row_dst(r)) & 15u) == 0;
        };
        for (int c = lane; c < 48; c += 32) {
            const int r = c / 6, piece = c - r * 6;
            if (row_vec(r))
                reinterpret_cast<double2 *>(row_dst(r))[piece] =
                    *reinterpret_cast<const double2 *>(&gst[r * 12 + piece * 2]);
        }
        if (valid && !row_vec(lane >> 2))
#pragma unroll
            for (int k = 0; k < 3; ++k) a.grad_total[i * 3 + k] = gst[lane * 3 + k];
    }
    if (is_last) {
        __shared__ double red[2 * (GT3 / 32)];
        gather_costs<GT3>(a, X.nt * Y.nt * Z.nt, nblk, false, size_t(a.n[0]) * a.n[1] * a.n[2], red);
    }
}

// ---------------------------------------------------------------------
// kernels: one pair (grid = tiles) and a batch of pairs (grid = work list
// of (pair, tile) items; pairs whose minimizer has finished are skipped)
// ---------------------------------------------------------------------
#ifndef MGR_WARP_MINB
#define MGR_WARP_MINB 3
#endif

template <int TZ, int COST>
__global__ void __launch_bounds__(NT3, MGR_WARP_MINB) k_warp3(const __grid_constant__ EvalArgs a)
{
    const int tile = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    warp3_body<TZ, COST, false>(a, blockIdx.x, blockIdx.y, blockIdx.z, tile);
}

template <int TZ>
__global__ void MGR_ADJ_BOUNDS k_adjoint3(EvalArgs a)
{
    const int tile = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    adjoint3_body<TZ>(a, blockIdx.x, blockIdx.y, blockIdx.z, tile);
}

__global__ void MGR_GATHER_BOUNDS k_gather3(EvalArgs a, int with_gradient, int image_from_dense)
{
    gather3_body(a, with_gradient, image_from_dense, blockIdx.x, gridDim.x);
}

// The NCC cost and force constants from the warp kernel's tile sums, one
// block of NT3 threads, so that the warp blocks end without a device-wide
// fence.  The adjoint kernel after it reads the
// constants.
__global__ void __launch_bounds__(NT3) k_finalise3(EvalArgs a)
{
    __shared__ double red[5 * (NT3 / 32)];
    pdl_wait();
    pdl_trigger();
    reduce_tile_sums(a, a.ax[0].nt * a.ax[1].nt * a.ax[2].nt, size_t(a.n[0]) * a.n[1] * a.n[2], red);
}

// the same for every running pair of a batch, a block each
__global__ void __launch_bounds__(NT3) k_finalise3_batch(const EvalArgs *__restrict__ args,
                                                         const int *__restrict__ active)
{
    __shared__ double red[5 * (NT3 / 32)];
    pdl_wait();
    pdl_trigger();
    if (!active[blockIdx.x]) return;
    const EvalArgs &a = args[blockIdx.x];
    reduce_tile_sums(a, a.ax[0].nt * a.ax[1].nt * a.ax[2].nt, size_t(a.n[0]) * a.n[1] * a.n[2], red);
}

__device__ __forceinline__ void decode_tile3(const EvalArgs &a, int t, int &bx, int &by, int &bz)
{
    const int ntx = a.ax[0].nt, nty = a.ax[1].nt;
    bx = t % ntx;
    by = (t / ntx) % nty;
    bz = t / (ntx * nty);
}

template <int TZ, int COST>
__global__ void __launch_bounds__(NT3, MGR_WARP_MINB) k_warp3_batch(const EvalArgs *__restrict__ args,
                                                                    const int2 *__restrict__ items,
                                                                    const int *__restrict__ active)
{
    const int2 it = items[blockIdx.x];
    pdl_wait();   // the minimizer sets the flags
    if (!active[it.x]) return;
    const EvalArgs &a = args[it.x];
    int bx, by, bz;
    decode_tile3(a, it.y, bx, by, bz);
    warp3_body<TZ, COST, true>(a, bx, by, bz, it.y);
}

template <int TZ>
__global__ void MGR_ADJ_BOUNDS k_adjoint3_batch(const EvalArgs *__restrict__ args,
                                                        const int2 *__restrict__ items, const int *__restrict__ active)
{
    const int2 it = items[blockIdx.x];
    pdl_wait();   // the minimizer sets the flags
    if (!active[it.x]) return;
    const EvalArgs &a = args[it.x];
    int bx, by, bz;
    decode_tile3(a, it.y, bx, by, bz);
    adjoint3_body<TZ>(a, bx, by, bz, it.y);
}

// Persistent forms of the batched warp and adjoint kernels: a grid of
// resident blocks draws (pair, tile) items from a device queue (queue[0],
// one atomic per item); the last block to finish resets the queue for the
// next launch (queue[1] counts finished blocks), so the launch can be
// replayed from a CUDA graph.
__device__ __forceinline__ bool next_item(int *queue, int nitems, const int2 *items, int2 &it, int &slot)
{
    __syncthreads();   // every thread is done with the previous item's shared memory
    if (threadIdx.x == 0) slot = atomicAdd(&queue[0], 1);
    __syncthreads();
    const int i = slot;
    if (i >= nitems) return false;
    it = items[i];
    return true;
}

__device__ __forceinline__ void queue_done(int *queue)
{
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&queue[1], 1) == int(gridDim.x) - 1) {
            queue[0] = 0;
            queue[1] = 0;
            __threadfence();
        }
    }
}

template <int TZ, int COST>
__global__ void __launch_bounds__(NT3, MGR_WARP_MINB) k_warp3_queue(const EvalArgs *__restrict__ args,
                                                                    const int2 *__restrict__ items, int nitems,
                                                                    const int *__restrict__ active, int *queue)
{
    __shared__ int slot;
    int2 it;
    pdl_wait();
    pdl_trigger();
    while (next_item(queue, nitems, items, it, slot)) {
        if (!active[it.x]) continue;
        const EvalArgs &a = args[it.x];
        int bx, by, bz;
        decode_tile3(a, it.y, bx, by, bz);
        warp3_body<TZ, COST, true>(a, bx, by, bz, it.y);
    }
    queue_done(queue);
}

template <int TZ>
__global__ void MGR_ADJ_BOUNDS k_adjoint3_queue(const EvalArgs *__restrict__ args,
                                                        const int2 *__restrict__ items, int nitems,
                                                        const int *__restrict__ active, int *queue)
{
    __shared__ int slot;
    int2 it;
    pdl_wait();
    pdl_trigger();
    while (next_item(queue, nitems, items, it, slot)) {
        if (!active[it.x]) continue;
        const EvalArgs &a = args[it.x];
        int bx, by, bz;
        decode_tile3(a, it.y, bx, by, bz);
        adjoint3_body<TZ>(a, bx, by, bz, it.y);
    }
    queue_done(queue);
}

__global__ void MGR_GATHER_BOUNDS k_gather3_batch(const EvalArgs *__restrict__ args,
                                                       const int2 *__restrict__ items, const int *__restrict__ active,
                                                       const int *__restrict__ nblocks)
{
    const int2 it = items[blockIdx.x];
    pdl_wait();   // the minimizer sets the flags
    if (!active[it.x]) return;
    gather3_body(args[it.x], 1, 0, it.y, nblocks[it.x]);
}

// float copy of the parameters (the warp and gather kernels read them as
// float, as the reference's spline evaluation does; FP64 conversions are
// slow on this GPU, so they are done once per evaluation).  It and
// k_params_host let the next kernel start without a wait of their own: they
// are only ever launched in plain stream order (launch_params_f32).
__global__ void __launch_bounds__(256) k_params_f32(const double *__restrict__ p, float *__restrict__ f, size_t n)
{
    pdl_trigger();   // the warp kernel may start its set-up (it waits for this kernel)
    for (size_t i = blockIdx.x * size_t(256) + threadIdx.x; i < n; i += size_t(gridDim.x) * 256) f[i] = float(p[i]);
}

// ---------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------
// The parameters read where the caller holds them (host memory that the
// device reads coherently): the device keeps a double and a float copy.  A
// non-finite value is stored as 0 in both and raises counters[7], so that
// the kernels after it run on finite parameters and the gather writes
// nothing to the caller's buffers.
__global__ void __launch_bounds__(256) k_params_host(const double *__restrict__ src, double *__restrict__ p,
                                                     float *__restrict__ f, size_t n, unsigned *__restrict__ bad)
{
    pdl_trigger();   // the warp kernel may start its set-up (it waits for this kernel)
    bool nonfinite = false;
    for (size_t i = blockIdx.x * size_t(256) + threadIdx.x; i < n; i += size_t(gridDim.x) * 256) {
        double v = src[i];
        if (!isfinite(v)) {
            nonfinite = true;
            v = 0.0;
        }
        p[i] = v;
        f[i] = float(v);
    }
    if (__any_sync(FULL, nonfinite) && (threadIdx.x & 31) == 0) atomicOr(bad, 1u);
}

void launch_params_f32(const EvalArgs &a, cudaStream_t st)
{
    const size_t n = size_t(a.nc[0]) * a.nc[1] * a.nc[2] * a.dim;
    const int nb = int(std::min<size_t>(1024, (n + 255) / 256));
    if (a.params_host)
        k_params_host<<<nb, 256, 0, st>>>(a.params_host, const_cast<double *>(a.params), a.params_f, n,
                                          a.counters + 7);
    else
        k_params_f32<<<nb, 256, 0, st>>>(a.params, a.params_f, n);
    count_launch();
}
size_t split3_smem(const EvalArgs &a, int which)
{
    const Axis &X = a.ax[0], &Y = a.ax[1], &Z = a.ax[2];
    if (which == 0)
        return size_t(3) * Z.fc * Y.fc * (X.fc + TX3) * sizeof(float) + size_t(RING_N) * RING_PLANE * sizeof(float);
    return (size_t(3) * Z.ac * TY3 * (TX3 + 1) +
            std::max(size_t(3) * Z.ac * TY3 * X.ac, size_t(AT3 / 32) * AD * AD_PLANE)) *
           sizeof(float);
}

namespace {

// the z-tile lengths the single-level kernels are compiled for:
// fn(std::integral_constant<int, TZ>{}) for the length tz, false when tz is
// not one of them.  The lengths between the powers of two let the
// autotuner fit a level's tiles to the waves of resident blocks: 128 planes
// in 20-plane tiles end with a row of 8-plane tiles that fills the last
// wave's gaps, where 16-plane tiles leave half of the last wave idle.
template <typename Fn>
bool with_tz(int tz, Fn &&fn)
{
    switch (tz) {
    case 4: fn(std::integral_constant<int, 4>{}); return true;
    case 8: fn(std::integral_constant<int, 8>{}); return true;
    case 12: fn(std::integral_constant<int, 12>{}); return true;
    case 16: fn(std::integral_constant<int, 16>{}); return true;
    case 20: fn(std::integral_constant<int, 20>{}); return true;
    case 24: fn(std::integral_constant<int, 24>{}); return true;
    case 32: fn(std::integral_constant<int, 32>{}); return true;
    default: return false;
    }
}

}  // namespace

bool tile_supported3(int tx, int ty, int tz)
{
    return tx == TX3 && ty == TY3 && with_tz(tz, [](auto) {});
}

// the batched and persistent kernels are compiled for the tile that the
// registration drivers run (registration_tile)
constexpr int BATCH_TZ = 16;

bool tile_supported3_batch(int tx, int ty, int tz)
{
    return tx == TX3 && ty == TY3 && tz == BATCH_TZ;
}

namespace {

template <int TZ, int COST>
void launch_warp3_zc(const EvalArgs &a, size_t sm, cudaStream_t st)
{
    raise_smem_limit(reinterpret_cast<const void *>(k_warp3<TZ, COST>), sm);
    launch_pdl(a.pdl != 0, k_warp3<TZ, COST>, dim3(a.ax[0].nt, a.ax[1].nt, a.ax[2].nt), dim3(NT3), sm, st, a);
}
template <int TZ>
void launch_warp3_z(const EvalArgs &a, size_t sm, cudaStream_t st)
{
    if (a.cost == MGR_COST_SSD)
        launch_warp3_zc<TZ, MGR_COST_SSD>(a, sm, st);
    else
        launch_warp3_zc<TZ, MGR_COST_NCC>(a, sm, st);
}

template <int TZ>
void launch_adjoint3_z(const EvalArgs &a, size_t sm, cudaStream_t st)
{
    raise_smem_limit(reinterpret_cast<const void *>(k_adjoint3<TZ>), sm);
    launch_pdl(a.pdl != 0, k_adjoint3<TZ>, dim3(a.ax[0].nt, a.ax[1].nt, a.ax[2].nt), dim3(AT3), sm, st, a);
}

}  // namespace

void launch_warp3(const EvalArgs &a, cudaStream_t st)
{
    launch_params_f32(a, st);
    const size_t sm = split3_smem(a, 0);
    with_tz(a.ax[2].t, [&](auto z) { launch_warp3_z<decltype(z)::value>(a, sm, st); });
    count_launch();
    if (!a.defer_cost || a.cost != MGR_COST_SSD) {
        launch_pdl(a.pdl != 0, k_finalise3, dim3(1), dim3(NT3), 0, st, a);
        count_launch();
    }
}

void launch_adjoint3(const EvalArgs &a, cudaStream_t st)
{
    const size_t sm = split3_smem(a, 1);
    with_tz(a.ax[2].t, [&](auto z) { launch_adjoint3_z<decltype(z)::value>(a, sm, st); });
    count_launch();
}

int gather3_blocks(const EvalArgs &a)
{
    return ((a.nc[0] + GBX - 1) / GBX) * ((a.nc[1] + GBY - 1) / GBY) * ((a.nc[2] + GBZ - 1) / GBZ);
}

void launch_gather3(const EvalArgs &a, int with_gradient, int dense, cudaStream_t st)
{
    launch_pdl(a.pdl != 0, k_gather3, dim3(gather3_blocks(a)), dim3(GT3), 0, st, a, with_gradient, dense);
    count_launch();
}

namespace {

// the batch's warp kernel by cost
auto warp3_batch_kernel(int cost)
{
    return cost == MGR_COST_SSD ? k_warp3_batch<BATCH_TZ, MGR_COST_SSD> : k_warp3_batch<BATCH_TZ, MGR_COST_NCC>;
}
auto warp3_queue_kernel(int cost)
{
    return cost == MGR_COST_SSD ? k_warp3_queue<BATCH_TZ, MGR_COST_SSD> : k_warp3_queue<BATCH_TZ, MGR_COST_NCC>;
}

}  // namespace

void prepare_split3_batch(int cost, size_t sm_warp, size_t sm_adj)
{
    raise_smem_limit(reinterpret_cast<const void *>(warp3_batch_kernel(cost)), sm_warp);
    raise_smem_limit(reinterpret_cast<const void *>(warp3_queue_kernel(cost)), sm_warp);
    raise_smem_limit(reinterpret_cast<const void *>(k_adjoint3_batch<BATCH_TZ>), sm_adj);
    raise_smem_limit(reinterpret_cast<const void *>(k_adjoint3_queue<BATCH_TZ>), sm_adj);
}

void launch_split3_batch(int cost, const EvalArgs *args, const int2 *items, int nitems, const int *active, size_t sm,
                         int which, bool pdl, cudaStream_t st)
{
    if (which == 0)
        launch_pdl(pdl, warp3_batch_kernel(cost), dim3(nitems), dim3(NT3), sm, st, args, items, active);
    else
        launch_pdl(pdl, k_adjoint3_batch<BATCH_TZ>, dim3(nitems), dim3(AT3), sm, st, args, items, active);
    count_launch();
}

// resident blocks of the persistent kernels (blocks per SM x SMs)
int split3_queue_grid(int cost, int which, size_t sm)
{
    int per_sm = 0;
    if (which == 0)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, warp3_queue_kernel(cost), NT3, sm);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_adjoint3_queue<BATCH_TZ>, AT3, sm);
    return std::max(1, per_sm) * device_sm_count();
}

void launch_split3_queue(int cost, const EvalArgs *args, const int2 *items, int nitems, const int *active, int *queue,
                         int grid, size_t sm, int which, bool pdl, cudaStream_t st)
{
    if (which == 0)
        launch_pdl(pdl, warp3_queue_kernel(cost), dim3(grid), dim3(NT3), sm, st, args, items, nitems, active, queue);
    else
        launch_pdl(pdl, k_adjoint3_queue<BATCH_TZ>, dim3(grid), dim3(AT3), sm, st, args, items, nitems, active, queue);
    count_launch();
}

void launch_finalise3_batch(const EvalArgs *args, int npairs, const int *active, bool pdl, cudaStream_t st)
{
    launch_pdl(pdl, k_finalise3_batch, dim3(npairs), dim3(NT3), 0, st, args, active);
    count_launch();
}

void launch_gather3_batch(const EvalArgs *args, const int2 *items, int nitems, const int *active, const int *nblocks,
                          bool pdl, cudaStream_t st)
{
    launch_pdl(pdl, k_gather3_batch, dim3(nitems), dim3(GT3), 0, st, args, items, active, nblocks);
    count_launch();
}

}  // namespace mgr

// Self-test of the bounded wait: one thread waits on phase 0 of an mbarrier
// that nothing arrives at (no copy is in flight), with the warp kernel's
// wait at a limit of SELFTEST_TRIES tries; it must give up and raise the
// flag, and the global timer (nanoseconds, independent of the SM clock)
// gives the time of one failed try.
namespace {
constexpr int SELFTEST_TRIES = 1024;

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__global__ void k_bounded_wait_selftest(unsigned *flag, long long *ns)
{
    __shared__ __align__(8) unsigned long long mb;
    const unsigned a = mgr::smem_u32(&mb);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(a) : "memory");
    const unsigned long long t0 = global_ns();
    if (!mgr::mbar_wait<SELFTEST_TRIES>(a, 0u)) atomicOr(flag, 1u);
    *ns = (long long)(global_ns() - t0);
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(a) : "memory");
}
}  // namespace

extern "C" mgr_status mgr_selftest_bounded_wait(int device, int *gave_up, double *us_per_try)
{
    if (!gave_up || !us_per_try) {
        mgr::set_last_error("mgr_selftest_bounded_wait: null argument");
        return MGR_ERR_ARG;
    }
    int prev = 0;
    cudaError_t e = cudaGetDevice(&prev);
    unsigned *flag = nullptr;
    long long *ns = nullptr;
    unsigned f = 0;
    long long t = 0;
    if (e == cudaSuccess) e = cudaSetDevice(device);
    if (e == cudaSuccess) e = mgr::dev_malloc(reinterpret_cast<void **>(&flag), sizeof(unsigned));
    if (e == cudaSuccess) e = mgr::dev_malloc(reinterpret_cast<void **>(&ns), sizeof(long long));
    if (e == cudaSuccess) e = cudaMemset(flag, 0, sizeof(unsigned));
    if (e == cudaSuccess) {
        k_bounded_wait_selftest<<<1, 1>>>(flag, ns);
        mgr::count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(&f, flag, sizeof f, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&t, ns, sizeof t, cudaMemcpyDeviceToHost);
    cudaFree(flag);
    cudaFree(ns);
    cudaSetDevice(prev);   // the caller's current device is left as it was
    if (e != cudaSuccess) {
        mgr::set_last_error(std::string("mgr_selftest_bounded_wait: ") + cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? MGR_ERR_OOM : MGR_ERR_CUDA;
    }
    *gave_up = f ? 1 : 0;
    *us_per_try = double(t) * 1e-3 / SELFTEST_TRIES;
    return MGR_OK;
}
