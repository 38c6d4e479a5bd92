"""Measured cases of the registration framework: what its users have it do,
through its public entry points, from one small 2D frame to a large volume.

  device   one cost+gradient evaluation with parameters and gradient on the
           GPU (Level.evaluate_device): the inner step of a device minimizer
  host     the same from host arrays (Level.evaluate_total): the inner step
           of a minimizer that runs on the host, as the library's own
           per-pair driver and the plugin adapter do
  value    the cost alone from host arrays (Level.value): line searches
  newpair  a new image pair on a kept level, then its first evaluation
           (Level.set_images_device, Level.evaluate_device)
  series   registration of a 2D perfusion series (register_batch_device)
  cohort   registration of 3D pairs of uneven size (register_batch_device)

Images are blob phantoms with noise, the moving one with displaced blobs
(and, for NCC, a smooth multiplicative bias), jointly normalised where the
registration driver would; parameters are spline coefficients in the middle
of a registration.
"""
import math

import numpy as np
import torch

import mia_gb300 as M
from mia_gb300 import registration as R

SERIES_SIZES = [(96, 96), (128, 112), (160, 144), (192, 160)]


def listed():
    return [
        # one small frame of a perfusion series: launches and latency
        dict(name="frame_96x96", kind="host", nx=96, ny=96, nz=0, rate=16.0, cost="ssd", weight=10.0, curl=1.0),
        # a large 2D slice
        dict(name="slice_1024x1024", kind="device", nx=1024, ny=1024, nz=0, rate=16.0, cost="ncc", weight=5.0,
             curl=1.0),
        # the coarsest level of a 3D cohort pair
        dict(name="coarse_40x44x36", kind="device", nx=40, ny=44, nz=36, rate=8.0, cost="ncc", weight=5.0, curl=1.0),
        # a volume of odd size on a fine grid, the curl part weighted apart
        dict(name="fine_121x143x109", kind="device", nx=121, ny=143, nz=109, rate=4.0, cost="ssd", weight=3.0,
             curl=0.3),
        # the benchmark pair, parameters on the device and on the host
        dict(name="pair_192x192x128", kind="device", nx=192, ny=192, nz=128, rate=8.0, cost="ssd", weight=10.0,
             curl=1.0),
        dict(name="host_192x192x128", kind="host", nx=192, ny=192, nz=128, rate=8.0, cost="ssd", weight=10.0,
             curl=1.0),
        # the multi-modal benchmark pair with a fine grid
        dict(name="ncc_256x256x256", kind="device", nx=256, ny=256, nz=256, rate=5.0, cost="ncc", weight=5.0,
             curl=1.0),
        # a large volume, ragged in every tile direction
        dict(name="large_383x351x317", kind="device", nx=383, ny=351, nz=317, rate=12.0, cost="ssd", weight=5.0,
             curl=1.0),
        # the cost alone at a cohort pair's full size
        dict(name="value_160x176x144", kind="value", nx=160, ny=176, nz=144, rate=8.0, cost="ncc", weight=5.0,
             curl=1.0),
        # new images on a kept level and their first evaluation
        dict(name="newpair_192x192x128", kind="newpair", nx=192, ny=192, nz=128, rate=8.0, cost="ssd", weight=10.0,
             curl=1.0),
        # a perfusion series, frames of four sizes
        dict(name="series_24", kind="series", npairs=24, rate=16.0, levels=2, maxiter=40, cost="ssd", weight=10.0),
        # a 3D cohort, pairs of uneven size
        dict(name="cohort_6", kind="cohort", npairs=6, lo=96, hi=176, rate=8.0, levels=3, maxiter=30, cost="ncc",
             weight=5.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "host", "host", "value", "newpair", "series", "cohort"])
    cost = rng.choice(["ssd", "ncc"])
    if kind == "series":
        return dict(kind=kind, npairs=rng.randint(4, 32), rate=rng.choice([12.0, 16.0]), levels=rng.randint(1, 2),
                    maxiter=rng.randint(15, 45), cost="ssd", weight=round(rng.uniform(2.0, 12.0), 2))
    if kind == "cohort":
        return dict(kind=kind, npairs=rng.randint(2, 6), lo=rng.randint(64, 96), hi=rng.randint(100, 160),
                    rate=rng.choice([8.0, 10.0]), levels=rng.randint(1, 2), maxiter=rng.randint(8, 25), cost=cost,
                    weight=round(rng.uniform(2.0, 12.0), 2))
    c = dict(kind=kind, cost=cost, weight=round(rng.uniform(1.0, 12.0), 2), curl=rng.choice([1.0, 1.0, 0.3, 2.0]))
    if rng.random() < 0.3:
        c.update(nx=_log(rng, 64, 1024), ny=_log(rng, 64, 1024), nz=0, rate=round(rng.uniform(6.0, 20.0), 1))
        return c
    while True:
        n = [_log(rng, 33, 400) for _ in range(3)]
        if n[0] * n[1] * n[2] <= 383 * 351 * 317:
            break
    # a fine grid on the smaller volumes only, as a registration would have it
    fine = 4.0 if n[0] * n[1] * n[2] < 1 << 24 else 8.0
    c.update(nx=n[0], ny=n[1], nz=n[2], rate=round(rng.uniform(fine, 12.0), 1))
    return c


def _size(case):
    return (case["nx"], case["ny"]) + ((case["nz"],) if case["nz"] else ())


def _csize(n, rate):
    """coefficients of one axis: floor((n - 1 + rate) / rate) in float, and the border"""
    return int((np.float32(n - 1) + np.float32(rate)) / np.float32(rate)) + 2


# ---------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------
def _images(size, seed, bias, normalise):
    """(moving, reference) float32 CUDA tensors [(z,) y, x]"""
    rng = np.random.default_rng(seed)
    dim, nb = len(size), 40 if len(size) == 3 else 12
    shape = size[::-1]
    centre = np.stack([rng.uniform(0, n, nb) for n in shape])
    sigma = rng.uniform(4.0, 16.0 if dim == 3 else 12.0, nb)
    amp = rng.uniform(50.0, 200.0, nb)
    shift = np.clip(rng.normal(0.0, 2.0, (dim, nb)), -4.0, 4.0)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    out = []
    for move in (shift, 0.0):
        lines = []
        for a, n in enumerate(shape):
            x = np.arange(n)[None, :] - (centre + move)[a][:, None]
            lines.append(torch.from_numpy(np.exp(-x * x / (2 * sigma[:, None] ** 2)).astype(np.float32)).cuda())
        lines[0] = lines[0] * torch.from_numpy(amp.astype(np.float32)).cuda()[:, None]
        rest = lines[1] if dim == 2 else (lines[1][:, :, None] * lines[2][:, None, :]).reshape(nb, -1)
        img = (lines[0].t() @ rest).reshape(shape)
        out.append(img + 2.0 * torch.randn(shape, generator=g, device="cuda"))
    mov, ref = out
    if bias:
        b = rng.normal(0.0, 0.1, (dim, 2))
        for a, n in enumerate(shape):
            t = np.linspace(-1.0, 1.0, n)
            f = torch.from_numpy(np.exp(b[a, 0] * t + b[a, 1] * t * t).astype(np.float32)).cuda()
            mov = mov * f.reshape([-1 if k == a else 1 for k in range(dim)])
    if normalise:
        both = torch.stack([mov, ref]).double()
        mean, sd = both.mean(), both.std()
        mov, ref = ((mov.double() - mean) / sd).float(), ((ref.double() - mean) / sd).float()
    return mov.contiguous(), ref.contiguous()


def _params(case, seed):
    """coefficients N(0, 1) clipped to +-2 voxels, smaller on grids finer than 8"""
    rng = np.random.default_rng(seed + 7)
    n = len(_size(case))
    for s in _size(case):
        n *= _csize(s, case["rate"])
    return np.clip(rng.normal(0.0, 1.0, n), -2.0, 2.0) * min(1.0, case["rate"] / 8.0)


def _pair_sizes(case):
    """the image sizes of a registration case (x, y[, z])"""
    if case["kind"] == "series":
        return [SERIES_SIZES[p % len(SERIES_SIZES)] for p in range(case["npairs"])]
    rng = np.random.default_rng(case["npairs"] + 1000 * case["lo"])
    return [tuple(int(v) for v in rng.integers(case["lo"], case["hi"] + 1, 3)) for _ in range(case["npairs"])]


def _pairs(case, seed):
    """raw (moving, reference) pairs of a registration case"""
    pairs = []
    for p, size in enumerate(_pair_sizes(case)):
        if case["kind"] == "series":
            mov, ref = _images(size, seed * 1009 + p, False, False)
            mov = (mov * (1.0 + 1.5 * math.sin(0.1 * p) ** 2)).contiguous()   # contrast passing through
        else:
            mov, ref = _images(size, seed * 1009 + p, True, False)
        pairs.append((mov, ref))
    return pairs


def prepare(case, seed):
    if case["kind"] in ("series", "cohort"):
        return dict(case=case, pairs=_pairs(case, seed), mz=R.minimizer("gsl", maxiter=case["maxiter"], step=0.1))
    mov, ref = _images(_size(case), seed, case["cost"] == "ncc", True)
    stream = torch.cuda.Stream()
    lv = M.Level(_size(case), rate=case["rate"], cost=case["cost"], penalty_weight=case["weight"], curl=case["curl"],
                 stream=stream.cuda_stream)
    p = _params(case, seed)
    torch.cuda.synchronize()
    lv.set_images_device(mov.data_ptr(), ref.data_ptr())
    s = dict(case=case, level=lv, stream=stream, params=p, grad=np.empty(lv.nparams))
    if case["kind"] in ("device", "newpair"):
        s["d_params"] = torch.from_numpy(p).cuda()
        s["d_grad"] = torch.empty(lv.nparams, dtype=torch.float64, device="cuda")
        s["d_costs"] = torch.empty(2, dtype=torch.float64, device="cuda")
    if case["kind"] == "newpair":
        s["mov"], s["ref"] = mov, ref
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("series", "cohort"):
        res = R.register_batch_device(s["pairs"], case["rate"], case["levels"], s["mz"], cost=case["cost"],
                                      penalty_weight=case["weight"])
        return dict(params=np.concatenate([r[0] for r in res]), csize=np.array([r[1] for r in res]),
                    cost=np.array([r[2] for r in res]), evaluations=np.array([r[3] for r in res]))
    lv = s["level"]
    if kind == "host":
        cost, grad = lv.evaluate_total(s["params"], grad_out=s["grad"])
        return dict(cost=cost, grad=grad)
    if kind == "value":
        image, penalty = lv.value(s["params"])
        return dict(image=image, penalty=penalty)
    if kind == "newpair":
        lv.set_images_device(s["mov"].data_ptr(), s["ref"].data_ptr())
    lv.evaluate_device(s["d_params"].data_ptr(), s["d_grad"].data_ptr(), s["d_costs"].data_ptr())
    return dict(costs=s["d_costs"], grad=s["d_grad"])


# ---------------------------------------------------------------------
# work
# ---------------------------------------------------------------------
def _eval_work(size, rate, grad):
    """one evaluation: both images and the parameters read once, the gradient
    written once; per voxel the spline's last axis, the interpolation's taps
    and weights, the cost, the force and the adjoint's first axis"""
    dim = len(size)
    n = float(np.prod(size))
    c = float(np.prod([_csize(s, rate) for s in size]))
    taps = 2 * 4 ** dim + 12 * dim + 8 * dim + 3
    stencil = (7 ** dim) * (18 if dim == 3 else 8)
    flops = n * (taps + (6 + 2 * dim + 8 * dim if grad else 0)) + c * stencil
    return 8.0 * n + 8.0 * dim * c * (2 if grad else 1), flops


def work(case):
    if case["kind"] in ("series", "cohort"):
        b = f = 0.0
        for size in _pair_sizes(case):
            for shift in range(case["levels"]):
                w = _eval_work([s >> shift for s in size], case["rate"], True)
                b += w[0] * (case["maxiter"] + 1)
                f += w[1] * (case["maxiter"] + 1)
        return {"bytes": b, "flops": f}
    b, f = _eval_work(_size(case), case["rate"], case["kind"] != "value")
    if case["kind"] == "newpair":
        n = float(np.prod(_size(case)))
        b, f = b + 8.0 * n, f + 8.0 * n * len(_size(case))   # both images in, the filtered one out
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------
def _bspline(t, p=0):
    """p-th derivative of the cubic B-spline"""
    a, sgn = np.abs(t), np.where(t < 0, -1.0, 1.0)
    r = np.maximum(2.0 - a, 0.0)
    inner = [(4.0 + a * a * (3.0 * a - 6.0)) / 6.0, sgn * a * (1.5 * a - 2.0), 3.0 * a - 2.0][p]
    outer = [r ** 3 / 6.0, -0.5 * sgn * r * r, r][p]
    return np.where(a <= 1.0, inner, outer)


def _apply(mats, x):
    """mats[a] (out x in, axis a of x counted from x-fastest) applied to every axis of x"""
    dim = x.dim()
    for a, m in enumerate(mats):
        x = torch.movedim(torch.tensordot(m, x, dims=([1], [dim - 1 - a])), 0, dim - 1 - a)
    return x


def _warp64(img, pos):
    """cubic B-spline interpolation of img at pos (components x first), mirror
    boundary, clamped to [min(0, min), max]"""
    shape = img.shape
    dim = len(shape)
    inv = []
    for n in shape[::-1]:
        a = np.zeros((n, n))
        for k in range(n):
            for d, w in ((-1, 1 / 6), (0, 4 / 6), (1, 1 / 6)):
                j = abs(k + d)
                a[k, j if j < n else 2 * n - 2 - j] += w
        inv.append(torch.from_numpy(np.linalg.inv(a)).cuda())
    coef = _apply(inv, img).reshape(-1)
    lo, hi = min(0.0, float(img.min())), float(img.max())
    out = torch.empty(img.numel(), dtype=torch.float64, device="cuda")
    flat = [p.reshape(-1) for p in pos]
    for at in range(0, out.numel(), 1 << 22):
        idx, wts = [], []
        for a in range(dim):
            n = shape[dim - 1 - a]
            p = flat[a][at:at + (1 << 22)]
            fl = torch.floor(p)
            f = p - fl
            w0, w3 = (1 - f) ** 3 / 6, f ** 3 / 6
            wts.append([w0, 1 - f - 2 * w0 + w3, f - 2 * w3 + w0, w3])
            ids = []
            for k in range(4):
                i = (fl.long() - 1 + k).abs() % (2 * n - 2)
                ids.append(torch.where(i < n, i, 2 * n - 2 - i))
            idx.append(ids)
        acc = 0.0
        for k in range(4 ** dim):
            w, i = 1.0, 0
            for a in range(dim - 1, -1, -1):
                j = (k >> (2 * a)) & 3
                w, i = w * wts[a][j], i * shape[dim - 1 - a] + idx[a][j]
            acc = acc + w * coef[i]
        out[at:at + (1 << 22)] = acc.clamp(lo, hi)
    return out.reshape(shape)


def _penalty64(case, csize, coefs):
    """(value, gradient) of the divcurl energy, the 1D integrals by Simpson's
    rule on 8 panels a knot interval (2D: inside the grid only)"""
    size = _size(case)
    dim = len(size)
    mats, scale = [], 1.0
    for n, nc in zip(size, csize):
        h = (nc - 1) / n
        scale /= h
        lo, hi = (0.0, float(nc)) if dim == 2 else (-4.0, nc + 4.0)
        x = np.linspace(lo, hi, int(hi - lo) * 16 + 1)
        w = np.full(x.size, 2.0)
        w[1::2] = 4.0
        w[0] = w[-1] = 1.0
        w /= 6.0 * 8.0
        j = np.arange(nc)
        b = [_bspline(x[:, None] - j, p) for p in range(3)]
        mats.append({(p, q): torch.from_numpy((b[p] * w[:, None]).T @ b[q] * h ** (p + q)).cuda()
                     for p in range(3) for q in range(3)})

    def block(c, cp):
        """the block's terms: (weight, orders at i, orders at j)"""
        def orders(a, b):
            o = [0] * dim
            o[a] += 1
            o[b] += 1
            return o
        if c == cp:
            t = [(1.0, orders(a, c), orders(a, c)) for a in range(dim)]
            return t + [(case["curl"], orders(a, b), orders(a, b)) for a in range(dim) for b in range(dim) if b != c]
        w = 2.0 * (1.0 - case["curl"])
        t = [(w, orders(a, c), orders(a, cp)) for a in range(dim)]
        if (c, cp) == (0, 1):
            t[-1] = (w, t[-1][2], t[-1][1])
        return [v for v in t if w]

    def times(c, cp, x):
        y = torch.zeros_like(x)
        for w, al, be in block(c, cp):
            y += scale * w * _apply([mats[a][al[a], be[a]] for a in range(dim)], x)
        return y

    value, grad = 0.0, []
    for c in range(dim):
        own = times(c, c, coefs[c])
        value += float((coefs[c] * own).sum())
        grad.append(2.0 * own)
    for c, cp in [(0, 1)] + ([(1, 2), (0, 2)] if dim == 3 else []):
        t = times(c, cp, coefs[cp])
        value += float((coefs[c] * t).sum())
        grad[c] += t
        grad[cp] += times(c, cp, coefs[c])
    return case["weight"] * value, [-case["weight"] * g for g in grad]


def exact(case, seed):
    if case["kind"] in ("series", "cohort"):
        return None   # many dependent steps: no value of its own
    size = _size(case)
    dim = len(size)
    csize = [_csize(n, case["rate"]) for n in size]
    mov, ref = (t.double() for t in _images(size, seed, case["cost"] == "ncc", True))
    # the spline sees its coefficients as float
    p = torch.from_numpy(_params(case, seed).astype(np.float32).astype(np.float64)).cuda()
    coefs = [p[c::dim].reshape(csize[::-1]) for c in range(dim)]
    W = []
    for n, nc in zip(size, csize):
        x = np.arange(n) * ((nc - 3) / (n - 1.0)) + 1.0
        W.append(torch.from_numpy(_bspline(x[:, None] - np.arange(nc)[None, :])).cuda())
    pos = []
    for c in range(dim):
        grid = torch.arange(size[c], dtype=torch.float64, device="cuda")
        pos.append(grid.reshape([-1 if k == dim - 1 - c else 1 for k in range(dim)]) - _apply(W, coefs[c]))
    wv = _warp64(mov, pos)
    if case["cost"] == "ssd":
        d = wv - ref
        image = 0.5 * float((d * d).sum())
        force = d
    else:
        a, b = wv - wv.mean(), ref - ref.mean()
        saa, sbb, sab = float((a * a).sum()), float((b * b).sum()), float((a * b).sum())
        image = 1.0 - sab * sab / (saa * sbb)
        force = 2.0 * sab / (saa * sbb) * (sab / saa * a - b)
    penalty, pgrad = _penalty64(case, csize, coefs)
    if case["kind"] == "value":
        return dict(image=image, penalty=penalty)
    grad = torch.empty_like(p)
    for c in range(dim):
        ax = dim - 1 - c
        g = torch.zeros_like(wv)
        n = size[c]
        g.narrow(ax, 1, n - 2).copy_(0.5 * (wv.narrow(ax, 2, n - 2) - wv.narrow(ax, 0, n - 2)))
        grad[c::dim] = (pgrad[c] - _apply([w.t().contiguous() for w in W], g * force)).reshape(-1)
    if case["kind"] == "host":
        return dict(cost=image + penalty, grad=grad.cpu().numpy())
    return dict(costs=torch.tensor([image, penalty], dtype=torch.float64), grad=grad)
