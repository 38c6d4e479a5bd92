"""The 2D split-path kernels at the sizes where their tiling can go wrong
(one below / at / above a tile, images smaller than one, grids finer and
coarser than a tile) for every tile shape, against the oracle; the forms of
launch and host access against one another, bit for bit.

Tolerances: the parity tests' own (tests/test_gpu_parity.py), cost 1e-5
relative and gradients 1e-4 relative L2 against the all-double oracle.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILES = [(32, 8), (32, 16), (64, 8), (64, 16), (32, 32)]
CASES = [((9, 7), 2.0), ((31, 33), 3.0), ((32, 32), 8.0), ((33, 31), 16.0), ((65, 17), 5.5), ((130, 64), 16.0),
         ((97, 129), 24.0)]


def _pair(size, seed):
    from mia_gb300 import synth
    ref = synth.blob_phantom(size[::-1], 8, sigma=(2.0, 5.0), seed=seed)
    mov = (np.roll(ref, 1, axis=1) * 1.1).astype(np.float32)
    return mov, ref


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("cost", ["ssd", "ncc"])
@pytest.mark.parametrize("size,rate", CASES)
def test_every_tile_against_the_oracle(size, rate, cost):
    import mia_gb300 as M
    from mia_gb300 import synth
    from oracle import oracle as O
    kw = dict(rate=rate, cost=cost, penalty_weight=2.0, curl=0.5)
    lv, o = M.Level(size, **kw), O.Level(size, precision=O.PREC_F64, **kw)
    mov, ref = _pair(size, 3)
    lv.set_images(mov, ref)
    o.set_images(mov, ref)
    p = synth.smooth_params(lv.csize, 1.5, seed=7)
    oi, op, ogi, ogp = o.evaluate(p)
    ov = o.value(p)
    for tile in TILES:
        lv.set_path("split", tile)
        ci, cp, gi, gp, gt = lv.evaluate(p)
        assert abs(ci - oi) <= 1e-5 * abs(oi) and abs(cp - op) <= 1e-5 * abs(op), tile
        assert _rel(gi, ogi) < 1e-4 and _rel(gp, ogp) < 1e-4, tile
        np.testing.assert_array_equal(gt, gi + gp)
        vi, vp = lv.value(p)
        assert abs(vi - ov[0]) <= 1e-5 * abs(ov[0]) and abs(vp - ov[1]) <= 1e-5 * abs(ov[1]), tile


@pytest.mark.parametrize("cost", ["ssd", "ncc"])
@pytest.mark.parametrize("size", [(61, 47), (192, 160)])
def test_host_access_and_launch_forms_agree(size, cost):
    """parameters and gradients in the caller's host memory, staged copies,
    device buffers, launches that overlap or not: the same bits; non-finite
    parameters are refused and nothing is written"""
    import torch

    import mia_gb300 as M
    from mia_gb300 import _lib
    from mia_gb300 import synth
    kw = dict(rate=9.0, cost=cost, penalty_weight=3.0)

    def level(env):
        os.environ.update(env)
        try:
            return M.Level(size, **kw)
        finally:
            for k in env:
                del os.environ[k]
    lvs = [level({}), level({"MGR_HOST_COPY": "1"}), level({"MGR_PDL": "0"})]
    mov, ref = _pair(size, 4)
    for lv in lvs:
        lv.set_images(mov, ref)
    for seed in (1, 2, 3):
        # the last one displaces past the mirror halo
        p = synth.smooth_params(lvs[0].csize, 1.5 if seed < 3 else 40.0, seed=seed)
        got = [lv.evaluate(p) for lv in lvs]
        for g in got[1:]:
            for x, y in zip(g, got[0]):
                assert np.array_equal(np.asarray(x), np.asarray(y))
        d_p = torch.from_numpy(p).cuda()
        d_g = torch.empty(lvs[0].nparams, dtype=torch.float64, device="cuda")
        d_c = torch.empty(2, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        lvs[0].evaluate_device(d_p.data_ptr(), d_g.data_ptr(), d_c.data_ptr())
        lvs[0].sync()
        assert np.array_equal(d_g.cpu().numpy(), got[0][4])
        assert d_c.cpu().tolist() == [got[0][0], got[0][1]]
    for lv in lvs:
        params, grad = synth.smooth_params(lv.csize, 1.0, seed=5), np.full(lv.nparams, 7.0)
        call = lv.bind_evaluate_total(params, grad)
        keep = params[lv.nparams - 1]
        params[lv.nparams - 1] = np.nan
        with pytest.raises(_lib.MgrError) as e:
            call()
        assert e.value.status == _lib.MGR_ERR_ARG and np.all(grad == 7.0)
        params[lv.nparams - 1] = keep
        c = call()
        w = lv.evaluate(params)
        assert c == w[0] + w[1] and np.array_equal(grad, w[4])


@pytest.mark.parametrize("at", [(16, 12), (31, 31), (32, 8), (8, 24), (33, 15)])
def test_an_infinite_force_reaches_the_four_coefficients_of_each_axis(at):
    """A force that overflows: the gradient is not finite at the four
    by four coefficients that the spline contracts its pixel with, those of
    weight 0 included (pixels on a coefficient), and finite at every other
    one, for every tile shape."""
    import mia_gb300 as M
    from mia_gb300 import synth
    size = (41, 33)   # rate 8: every eighth pixel lies on a coefficient
    rng = np.random.default_rng(5)
    mov, ref = (1e6 * rng.random((2, size[1], size[0]))).astype(np.float32)
    ref[at[1], at[0]] = 3e38   # times a difference of about 1e5
    lv = M.Level(size, rate=8.0, cost="ssd")
    p = synth.smooth_params(lv.csize, 0.7, seed=2)
    ncx, ncy = lv.csize[:2]

    def first(i):   # first coefficient o >= 0 with |i / 8 + 1 - o| < 2
        return i // 8
    want = np.zeros((ncy, ncx), bool)
    want[first(at[1]):first(at[1]) + 4, first(at[0]):first(at[0]) + 4] = True
    lv.set_images(mov, ref)
    for tile in TILES:
        lv.set_path("split", tile)
        g = np.asarray(lv.evaluate(p)[2]).reshape(ncy, ncx, 2)
        np.testing.assert_array_equal(~np.isfinite(g).all(axis=2), want, err_msg=str(tile))


# grids with several coefficients per voxel, up to windows of four that leave
# coefficients out between them (five per voxel)
@pytest.mark.parametrize("cost", ["ssd", "ncc"])
@pytest.mark.parametrize("size,csize", [((8, 16), (40, 80)), ((9, 7), (45, 10)), ((33, 20), (110, 62)),
                                        ((40, 33), (163, 130))])
def test_grids_finer_than_the_voxels(size, csize, cost):
    import mia_gb300 as M
    from mia_gb300 import synth
    from oracle import oracle as O
    kw = dict(csize=csize, cost=cost)
    lv, o = M.Level(size, **kw), O.Level(size, precision=O.PREC_F64, **kw)
    mov, ref = _pair(size, 3)
    lv.set_images(mov, ref)
    o.set_images(mov, ref)
    p = synth.smooth_params(lv.csize, 1.0, seed=7)
    oi, _, ogi, _ = o.evaluate(p)
    for tile in TILES:
        lv.set_path("split", tile)
        ci, _, gi, _, _ = lv.evaluate(p)
        assert abs(ci - oi) <= 1e-5 * abs(oi) and _rel(gi, ogi) < 1e-4, tile
