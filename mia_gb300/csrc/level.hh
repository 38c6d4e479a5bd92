// level.hh — the per-level state behind an mgr_level handle (device
// buffers, tables, stream); shared by the C ABI and the batched driver.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "../../include/mgr.h"
#include "mgr_kernels.hh"
#include "tables.hh"
#include "tune.hh"

namespace mgr {

struct CudaError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
struct StateError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
// a bounded device wait gave up (the kernel raised the level's status flag)
struct TimeoutError : std::runtime_error {
    using std::runtime_error::runtime_error;
};

inline void ck(cudaError_t e, const char *what)
{
    if (e != cudaSuccess) {
        std::string m = std::string(what) + ": " + cudaGetErrorString(e);
        if (e == cudaErrorMemoryAllocation) throw std::bad_alloc();
        throw CudaError(m);
    }
}

// Keep freed stream-ordered allocations of `device` cached in its default
// memory pool (up to a bound) so that repeated level setup does not map and
// unmap device memory.
void configure_pool(int device);

// Device buffer in stream-ordered memory: allocated on and freed on the
// stream given to alloc(), which must outlive the buffer.  Growing keeps the
// old contents only when the old allocation is large enough.
template <class T>
struct DevBuf {
    T *p = nullptr;
    size_t n = 0;
    cudaStream_t st = nullptr;
    bool own = true;   // false: part of another buffer (borrow)
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() { release(); }
    void release()
    {
        if (p && own) cudaFreeAsync(p, st);
        p = nullptr;
        n = 0;
        own = true;
    }
    // count elements at q, inside a buffer that outlives this one
    void borrow(void *q, size_t count)
    {
        release();
        p = static_cast<T *>(q);
        n = count;
        own = false;
    }
    void swap(DevBuf &o) noexcept
    {
        std::swap(p, o.p);
        std::swap(n, o.n);
        std::swap(st, o.st);
        std::swap(own, o.own);
    }
    void alloc(size_t count, cudaStream_t s)
    {
        if (count <= n && p) return;
        release();
        if (count == 0) return;
        ck(dev_malloc_async(reinterpret_cast<void **>(&p), count * sizeof(T), s), "cudaMallocAsync");
        st = s;
        n = count;
    }
    void upload(const std::vector<T> &h, cudaStream_t s)
    {
        alloc(h.size(), s);
        if (!h.empty()) ck(cudaMemcpyAsync(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s), "upload");
    }
};

// The buffers that `each` lists (each(f) calls f(buffer, count) for all of
// them) in one allocation: a level has about twenty, and the cost of a
// stream-ordered allocation grows with the blocks that the pool holds and the
// streams they were freed on.  The slab is a fresh one: buffers that borrow
// from another slab keep it until this one has its memory.
template <class Each>
void alloc_together(DevBuf<unsigned char> &slab, cudaStream_t s, Each each)
{
    auto bytes = [](auto &b, size_t count) { return (count * sizeof(*b.p) + 255) & ~size_t(255); };
    size_t total = 0;
    each([&](auto &b, size_t count) { total += bytes(b, count); });
    slab.alloc(total, s);
    size_t at = 0;
    each([&](auto &b, size_t count) {
        if (count == 0) b.release();
        else b.borrow(slab.p + at, count);
        at += bytes(b, count);
    });
}

// the per-axis tables of a level, packed with the other tables into one
// host blob and uploaded with one copy; `off` are byte offsets into it
struct AxisDev {
    AxisHost h;
    size_t off[11] = {};   // fs, as, rows, ftile0, atile0, gtile, fw, aw, glist, glen, win
    const unsigned char *base = nullptr;

    template <class T>
    static size_t pack(std::vector<unsigned char> &blob, const std::vector<T> &v)
    {
        const size_t o = (blob.size() + 255) & ~size_t(255);
        blob.resize(o + v.size() * sizeof(T));
        if (!v.empty()) std::memcpy(blob.data() + o, v.data(), v.size() * sizeof(T));
        return o;
    }
    void pack_all(std::vector<unsigned char> &blob)
    {
        off[0] = pack(blob, h.fs);
        off[1] = pack(blob, h.as);
        off[2] = pack(blob, h.rows);
        off[3] = pack(blob, h.ftile0);
        off[4] = pack(blob, h.atile0);
        off[5] = pack(blob, h.gtile);
        off[6] = pack(blob, h.fw);
        off[7] = pack(blob, h.aw);
        off[8] = pack(blob, h.glist);
        off[9] = pack(blob, h.glen);
        off[10] = pack(blob, h.win);
    }
    Axis view() const
    {
        Axis a;
        a.fs = reinterpret_cast<const int *>(base + off[0]);
        a.as = reinterpret_cast<const int *>(base + off[1]);
        a.rows = reinterpret_cast<const int2 *>(base + off[2]);
        a.ftile0 = reinterpret_cast<const int *>(base + off[3]);
        a.atile0 = reinterpret_cast<const int *>(base + off[4]);
        a.gtile = reinterpret_cast<const int2 *>(base + off[5]);
        a.fw = reinterpret_cast<const float4 *>(base + off[6]);
        a.aw = reinterpret_cast<const float4 *>(base + off[7]);
        a.glist = reinterpret_cast<const int *>(base + off[8]);
        a.glen = reinterpret_cast<const int *>(base + off[9]);
        a.win = reinterpret_cast<const int2 *>(base + off[10]);
        a.n = h.n;
        a.nc = h.nc;
        a.t = h.t;
        a.nt = h.nt;
        a.fc = h.fc;
        a.ac = h.ac;
        return a;
    }
};

}  // namespace mgr

using namespace mgr;

struct mgr_level {
    mgr_level_desc d{};
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int n[3] = {1, 1, 1}, nc[3] = {1, 1, 1};
    size_t N = 0, ncoef = 0, nparams = 0;
    int path = MGR_PATH_SPLIT;
    int tile[3] = {32, 8, 16};
    AxisDev ax[3];
    // the allocations that hold the buffers below: images, state (counters,
    // scalars), and what depends on the coefficient grid and the tile
    DevBuf<unsigned char> slab_images, slab_state, slab_grid;
    DevBuf<unsigned char> axis_tables;   // the packed AxisDev tables, then the penalty's
    std::vector<float> ptable_host;                        // 3D: the penalty's cells
    std::shared_ptr<const Penalty2Table> penalty2_host;    // 2D
    // MGR_PATH_FUSED: the tables of the fused kernel's tiles (30 x 8 x TZ),
    // for its launch and the gather after it; the other kernels keep ax
    AxisDev axf[3];
    DevBuf<unsigned char> axis_tables_f;
    int slot_f = 0;
    DevBuf<float> coef, coef_pad, ref, warped, minmax, partial, ptable, pen_val, params_f;
    DevBuf<float2> mmpart;
    DevBuf<double> params, grad_total, grad_image, grad_penalty, scalars, costs, tile_sums, pen_part, means, mpart;
    DevBuf<unsigned int> counters;
    DevBuf<int> pen_rowptr, pen_col;
    DevBuf<float> grid, force, tmp1, tmp2;   // plain path and standalone force/translate
    // (rebind() below lists every DevBuf member)
    CUtensorMap tmap{};     // 3D: tensor map of coef_pad
    bool has_tmap = false;
    int slot = 0;
    bool images_set = false;
    bool timing = false;
    // 1: events around every kernel (launched one after another); 2: events
    // around the whole evaluation only (kernels overlap as in untimed runs)
    int timing_mode = 0, ev_mode = 0;
    // a deferred cost finalisation (EvalArgs::defer_cost) is possible
    bool can_defer() const { return d.dim == 3 || d.cost == MGR_COST_SSD; }
    // programmatic dependent launch of the split path's kernels (MGR_PDL=0
    // in the environment at level creation turns it off)
    bool pdl = true;
    // the device reads and writes the caller's host memory in place
    // (coherent_host_access): evaluate moves parameters, gradient and costs
    // with the kernels' own loads and stores instead of staged copies
    bool coherent = false;
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
    bool ev_recorded = false;
    // move the level to stream s: its later work and the stream-ordered
    // frees of all its buffers go to s (the caller has ordered s after the
    // work queued on the old stream)
    void rebind(cudaStream_t s)
    {
        if (own_stream) throw std::invalid_argument("a level with its own stream cannot be moved");
        stream = s;
        auto re = [s](auto &b) {
            if (b.p) b.st = s;
        };
        re(slab_images), re(slab_state), re(slab_grid);
        re(axis_tables);
        re(axis_tables_f);
        re(coef), re(coef_pad), re(ref), re(warped), re(minmax), re(partial), re(ptable), re(pen_val), re(params_f);
        re(mmpart);
        re(params), re(grad_total), re(grad_image), re(grad_penalty), re(scalars), re(costs), re(tile_sums);
        re(pen_part), re(means), re(mpart);
        re(counters);
        re(pen_rowptr), re(pen_col);
        re(grid), re(force), re(tmp1), re(tmp2);
    }
    void record(int k)
    {
        if (timing && (timing_mode == 1 || k == 0 || k == 3)) ck(cudaEventRecord(ev[k], stream), "cudaEventRecord");
    }
    // 4 doubles of pinned host memory for small read-backs (costs, status)
    double *host_small_p = nullptr;
    double *host_small()
    {
        if (!host_small_p) ck(host_malloc_pinned(reinterpret_cast<void **>(&host_small_p), 4 * sizeof(double)),
                              "cudaMallocHost");
        return host_small_p;
    }
    ~mgr_level()
    {
        for (auto &e : ev)
            if (e) cudaEventDestroy(e);
        if (host_small_p) cudaFreeHost(host_small_p);
    }

    // a level made on another level's images (the refine pass of a batched
    // registration level): the image buffers are that level's, which
    // outlives this one; only one of the two is evaluated at a time
    const mgr_level *images_from = nullptr;

    // the kernels' arguments; `fused`: with the fused kernel's tile tables
    EvalArgs args(bool fused = false) const
    {
        const mgr_level &I = images_from ? *images_from : *this;
        EvalArgs a{};
        a.tmap = I.tmap;
        a.has_tmap = I.has_tmap;
        a.dim = d.dim;
        for (int k = 0; k < 3; ++k) {
            a.n[k] = n[k];
            a.nc[k] = nc[k];
            a.ax[k] = fused ? axf[k].view() : ax[k].view();
        }
        a.coef_img = I.coef.p;
        a.coef_pad = I.coef_pad.p;
        a.pad_rows = n[1] + 2 * PAD_H;
        a.ref = I.ref.p;
        a.warped = I.warped.p;
        a.minmax = I.minmax.p;
        a.params = params.p;
        a.params_f = params_f.p;
        a.convert = d.dim == 2;
        a.cost = d.cost;
        a.ssd_norm = d.ssd_norm;
        a.cost_weight = d.cost_weight;
        a.centers = I.means.p;
        a.partial = partial.p;
        a.slot = fused ? slot_f : slot;
        a.tile_sums = tile_sums.p;
        a.counters = counters.p;
        a.pdl = pdl && timing_mode != 1;
        a.scalars = scalars.p;
        a.has_penalty = d.has_penalty;
        double prod = double(d.size[0]) * d.size[1] * (d.dim == 3 ? d.size[2] : 1);
        a.pen_weight = d.pen_norm ? d.pen_weight / double(float(prod)) : d.pen_weight;
        a.pen_grad_w = (d.pen_corrected ? 1.0 : -1.0) * a.pen_weight;
        a.pen_grad_wf = float(a.pen_grad_w);
        a.cost_wf = float(a.cost_weight);
        a.ptable = ptable.p;
        a.pen_rowptr = pen_rowptr.p;
        a.pen_col = pen_col.p;
        a.pen_val = reinterpret_cast<const float4 *>(pen_val.p);
        a.pen_part = pen_part.p;
        a.grad_total = grad_total.p;
        a.grad_image = nullptr;
        a.grad_penalty = nullptr;
        a.costs = costs.p;
        return a;
    }

    // whether tile t is compiled in and, in 3D, its blocks' shared memory
    // fits on a grid of g coefficients: `strict`, the warp block three to an SM and the adjoint block in
    // 64 KiB (the rule without measurements); else what a launch allows
    // (the autotuner measured the shape, occupancy included)
    bool tile_fits(const int g[3], const int t[3], bool strict = true) const
    {
        if (!tile_supported(d.dim, t[0], t[1], t[2])) return false;
        if (d.dim == 2) return true;
        AxisHost hx, hy, hz;
        build_axis(hx, n[0], g[0], t[0]);
        build_axis(hy, n[1], g[1], t[1]);
        build_axis(hz, n[2], g[2], t[2]);
        const size_t w =
            (size_t(3) * hz.fc * hy.fc * (hx.fc + 32) + 32 + size_t(WARP_RING_PLANES) * 16 * 64) * sizeof(float);
        // (split3_smem(a, 1) but for the adjoint's ring, which takes at most
        // 17 KB more, and none where its windows are that large)
        const size_t adj = size_t(3) * hz.ac * 8 * (33 + hx.ac) * sizeof(float);
        if (strict) return w <= 74 * 1024 && adj <= 64 * 1024;
        return w + 128 <= 200 * 1024 && adj <= 200 * 1024;
    }

    // the tile for a grid of g coefficients into t: that of the autotuner's
    // nearest case (tune.cc) when a launch allows it, else 32x16 in 2D and in
    // 3D the deepest z tile (16, 8, 4) that fits three warp blocks to an SM
    void choose_tile(const int g[3], int t[3]) const
    {
        if (tuned_tile(d.dim, n, g, t) && tile_fits(g, t, false)) return;
        t[0] = 32;
        t[1] = d.dim == 3 ? 8 : 16;
        t[2] = 1;
        if (d.dim == 2) return;
        static const int tzs[3] = {16, 8, 4};
        for (int z : tzs) {
            t[2] = z;
            if (tile_fits(g, t)) return;
        }
    }

    // the per-axis tables of tiles t on a grid of g coefficients into A,
    // packed at the end of blob; returns the number of tiles and sets the
    // partial slot size
    int build_axis_set(const int g[3], const int t[3], AxisDev (&A)[3], std::vector<unsigned char> &blob,
                       int &slot_size) const
    {
        const int D = d.dim;
        AxisDev *ax = A;
        for (int k = 0; k < D; ++k) build_axis(ax[k].h, n[k], g[k], t[k]);
        {
            // per axis and coefficient: the partial-slot offset parts of the
            // tiles that hold it, slot entry (tx, ty[, tz]) of coefficient
            // (cx, cy[, cz]) being at glist_x + glist_y [+ glist_z]
            const int acz = D == 3 ? ax[2].h.ac : 1, ntz = D == 3 ? ax[2].h.nt : 1;
            const int sl = D * ax[0].h.ac * ax[1].h.ac * acz;
            const long long total = (long long)ax[0].h.nt * ax[1].h.nt * ntz * sl;
            const long long ts[3] = {sl, (long long)ax[0].h.nt * sl, (long long)ax[0].h.nt * ax[1].h.nt * sl};
            const long long ls[3] = {D, (long long)ax[0].h.ac * D, (long long)ax[0].h.ac * ax[1].h.ac * D};
            for (int k = 0; k < D; ++k) {
                AxisHost &h = ax[k].h;
                h.glist.assign(size_t(h.nc) * GATHER_LMAX, 0);
                h.glen.assign(h.nc, -1);
                for (int c = 0; c < h.nc; ++c) {
                    const int lo = h.gtile[size_t(c) * 2], hi = h.gtile[size_t(c) * 2 + 1];
                    const int cnt = std::max(hi - lo + 1, 0);
                    if (cnt > GATHER_LMAX || total >= (1LL << 31)) continue;
                    for (int j = 0; j < cnt; ++j)
                        h.glist[size_t(c) * GATHER_LMAX + j] =
                            int((lo + j) * ts[k] + (c - h.atile0[lo + j]) * ls[k]);
                    h.glen[c] = cnt;
                }
            }
        }
        for (int k = 0; k < D; ++k) ax[k].pack_all(blob);
        slot_size = D * ax[0].h.ac * ax[1].h.ac * (D == 3 ? ax[2].h.ac : 1);
        return ax[0].h.nt * ax[1].h.nt * (D == 3 ? ax[2].h.nt : 1);
    }

    // Moves the level to a grid of g coefficients, the split path's tile t and
    // a path: the tables (with the penalty's, one upload), the parameter and
    // gradient buffers and the partials.  All that can fail comes first and
    // leaves the level as it was; then the new state takes the old one's
    // place.  It is a fresh allocation: kernels queued earlier may still read
    // the old one, which is freed in stream order.
    void reshape(const int g[3], const int t[3], int new_path)
    {
        const int D = d.dim;
        AxisDev A[3], AF[3];
        std::vector<unsigned char> blob, blob_f;
        int sl = 0, sl_f = 0;
        const int ntiles = build_axis_set(g, t, A, blob, sl);
        size_t part = size_t(ntiles) * sl, sums = size_t(ntiles);
        if (new_path == MGR_PATH_FUSED) {
            // (its footprints count on it)
            for (int k = 0; k < D; ++k)
                if (g[k] - 3 > n[k] - 1)
                    throw std::invalid_argument("the fused path needs a coefficient spacing of at least one voxel");
            // the fused kernel's tile: 30 interior voxels in x (32 lanes with
            // the halo), 8 rows, the level's z tile
            const int tf[3] = {30, 8, t[2]};
            const int ntf = build_axis_set(g, tf, AF, blob_f, sl_f);
            part = std::max(part, size_t(ntf) * sl_f);
            sums = std::max(sums, size_t(ntf));
        }
        // the penalty's cells (3D: translation-invariant; 2D:
        // boundary-clipped CSR rows, cached across levels of equal grid)
        const bool new_grid = !slab_grid.p || g[0] != nc[0] || g[1] != nc[1] || g[2] != nc[2];
        std::vector<float> cells3;
        std::shared_ptr<const Penalty2Table> cells2 = penalty2_host;
        if (d.has_penalty && new_grid) {
            const float range[3] = {float(d.size[0]), float(d.size[1]), float(D == 3 ? d.size[2] : 1)};
            if (D == 3) cells3 = build_penalty3(g, range, d.pen_div, d.pen_curl);
            else cells2 = penalty2_cached(g, range, d.pen_div, d.pen_curl);
        }
        const std::vector<float> &p3 = new_grid ? cells3 : ptable_host;
        // 2D cells are many on large grids (49 per coefficient, 20 bytes each):
        // from 256 KB on they are uploaded from the cached table as it is, as
        // packing them costs more than the three uploads it saves.  A level
        // made with them packed / apart: 88 / 93 us at 165 KB (192x160, rate
        // 16), 115 / 116 at 318 KB, 176 / 154 at 714 KB, 637 / 385 at 4.3 MB
        // (1024x1024)
        const bool apart = d.has_penalty && D == 2 && cells2->col.size() * 20 >= 256 * 1024;
        size_t at_pen[3] = {0, 0, 0};
        if (d.has_penalty && D == 3) {
            at_pen[0] = AxisDev::pack(blob, p3);
        } else if (d.has_penalty && !apart) {
            at_pen[0] = AxisDev::pack(blob, cells2->rowptr);
            at_pen[1] = AxisDev::pack(blob, cells2->col);
            at_pen[2] = AxisDev::pack(blob, cells2->val);
        }
        EvalArgs sizes{};   // what the counts below depend on
        sizes.dim = D;
        for (int k = 0; k < 3; ++k) sizes.nc[k] = g[k];
        const size_t ncoefs = size_t(g[0]) * g[1] * g[2], np = ncoefs * D, plain_blocks = (N + 255) / 256;
        struct {
            DevBuf<unsigned char> slab, tables, tables_f;
            DevBuf<double> params, grad_total, tile_sums, pen_part;
            DevBuf<float> params_f, partial, pen_val;
            DevBuf<int> pen_rowptr, pen_col;
        } to;
        alloc_together(to.slab, stream, [&](auto buf) {
            buf(to.params, np);
            buf(to.params_f, np);
            buf(to.grad_total, np);
            buf(to.tables, blob.size());
            buf(to.partial, part);
            buf(to.tile_sums, std::max<size_t>(sums, plain_blocks) * 5);
            buf(to.pen_part, size_t(gather_blocks(sizes)) + 1);
            buf(to.pen_rowptr, apart ? cells2->rowptr.size() : 0);
            buf(to.pen_col, apart ? cells2->col.size() : 0);
            buf(to.pen_val, apart ? cells2->val.size() : 0);
        });
        to.tables.upload(blob, stream);
        if (apart) {
            to.pen_rowptr.upload(cells2->rowptr, stream);
            to.pen_col.upload(cells2->col, stream);
            to.pen_val.upload(cells2->val, stream);
        }
        to.tables_f.upload(blob_f, stream);

        // nothing fails from here on
        slab_grid.swap(to.slab);
        params.swap(to.params);
        params_f.swap(to.params_f);
        grad_total.swap(to.grad_total);
        axis_tables.swap(to.tables);
        axis_tables_f.swap(to.tables_f);
        partial.swap(to.partial);
        tile_sums.swap(to.tile_sums);
        pen_part.swap(to.pen_part);
        for (int k = 0; k < 3; ++k) {
            A[k].base = axis_tables.p;
            AF[k].base = axis_tables_f.p;
            ax[k] = std::move(A[k]);
            axf[k] = std::move(AF[k]);
            nc[k] = g[k];
            tile[k] = t[k];
        }
        slot = sl;
        slot_f = sl_f;
        ncoef = ncoefs;
        nparams = np;
        path = new_path;
        if (new_grid) ptable_host = std::move(cells3);
        penalty2_host = std::move(cells2);
        if (apart) {
            pen_rowptr.swap(to.pen_rowptr);
            pen_col.swap(to.pen_col);
            pen_val.swap(to.pen_val);
        } else if (d.has_penalty && D == 3) {
            ptable.borrow(axis_tables.p + at_pen[0], ptable_host.size());
        } else if (d.has_penalty) {
            pen_rowptr.borrow(axis_tables.p + at_pen[0], penalty2_host->rowptr.size());
            pen_col.borrow(axis_tables.p + at_pen[1], penalty2_host->col.size());
            pen_val.borrow(axis_tables.p + at_pen[2], penalty2_host->val.size());
        }
    }

    // counters and scalars, zero; means of the images
    void alloc_state()
    {
        alloc_together(slab_state, stream, [&](auto buf) {
            buf(counters, 8);
            buf(scalars, SC_NSLOTS);
            buf(costs, 2);
            buf(means, 2);
        });
        ck(cudaMemsetAsync(slab_state.p, 0, slab_state.n, stream), "memset");
    }
};

namespace mgr {
// The tile of the registration drivers' split path, per pair (register.cu)
// and batched (batch.cu), so that both run the same kernels in the same
// order: 32x8x16 in 3D, 32x16 in 2D (but for the last bits of a 3D SSD tile
// that does not fit the tap ring, warp3_body's BATCH).  The autotuner's table
// times single evaluations, where the tile sets the latency of one launch; in
// the batch every launch carries all pairs and the deeper tile's lower
// per-item overhead wins (60-frame 2D series: 1733-1778 pairs/s with 32x16
// against 1389-1415 with the tuned 32x8; the 3D cohort the same either way).
inline void registration_tile(int dim, int t[3])
{
    t[0] = 32;
    t[1] = dim == 3 ? 8 : 16;
    t[2] = dim == 3 ? 16 : 1;
}
// mgr_level_create, with the split path's tile when tile is given (and fits,
// by the strict rule or not: else the level keeps the one it would choose)
mgr_status level_create(const mgr_level_desc *desc, int device, void *stream, const int *tile, bool strict,
                        mgr_level **out);
// mgr_level_set_images_device without the final stream synchronisation
void level_set_images_async(mgr_level *L, const float *d_src, const float *d_ref);
// a new coefficient grid (and tile) on a level, images kept
void level_set_grid(mgr_level *L, const int csize[3], const int tile[3]);
// a level with the coefficient grid csize on the images of level S (same
// sizes, cost, penalty, path and tile; S must outlive it), made on stream st
mgr_level *level_create_on_images(const mgr_level *S, const int csize[3], cudaStream_t st);
}  // namespace mgr

namespace mgr {
// True when the device reads and writes pageable host memory coherently,
// translating through the host's page tables (Grace-based systems such as
// GB300, where the CPU-GPU link is cache coherent), unless the environment
// variable MGR_HOST_COPY is set to a value other than 0 (staged copies).
inline bool coherent_host_access(int device)
{
    int pageable = 0, host_tables = 0;
    const char *force_copy = std::getenv("MGR_HOST_COPY");
    bool ok = cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, device) == cudaSuccess &&
              cudaDeviceGetAttribute(&host_tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables, device) ==
                  cudaSuccess;
    cudaGetLastError();
    return ok && pageable == 1 && host_tables == 1 && !(force_copy && *force_copy && *force_copy != '0');
}

// Queue a read of the level's device status flag (counters[6], raised by a
// kernel whose bounded wait gave up) into *flag; after the stream has been
// synchronised, throw_if_flagged clears it and throws TimeoutError.
inline void read_status_flag(mgr_level *L, unsigned *flag)
{
    ck(cudaMemcpyAsync(flag, L->counters.p + 6, sizeof(unsigned), cudaMemcpyDeviceToHost, L->stream), "status D2H");
}
inline void throw_if_flagged(mgr_level *L, unsigned flag)
{
    if (flag) {
        ck(cudaMemsetAsync(L->counters.p + 6, 0, sizeof(unsigned), L->stream), "status reset");
        throw TimeoutError("a bounded device wait gave up (bulk copy did not complete)");
    }
}
}  // namespace mgr
