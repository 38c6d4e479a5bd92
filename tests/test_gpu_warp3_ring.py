"""The 3D warp kernel's walk where it can go wrong: tiles whose last step has
one plane, one plane in all, taps that just fit the shared-memory ring, just
do not, or leave the padded copy, and displacements that are not numbers.

Tolerance: as for every warped image (tests/test_gpu_parity.py), 1e-5 of the
largest value against the oracle at reference precision, costs 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _level(size, rate, cost):
    import mia_gb300 as M
    from mia_gb300 import synth
    ref = synth.blob_phantom(size[::-1], 10, sigma=(4.0, 8.0), seed=4)
    mov = np.roll(ref, 2, axis=2).astype(np.float32)
    lv = M.Level(size, rate=rate, cost=cost, penalty_weight=1.0)
    lv.set_images(mov, ref)
    return lv, mov, ref


@pytest.mark.parametrize("size", [(40, 33, 21), (33, 9, 33), (70, 16, 13)])
@pytest.mark.parametrize("amplitude", [0.0, 1.0, 4.0, 8.0, 14.0, 30.0])
def test_walk_against_the_oracle(size, amplitude):
    from oracle import oracle as O
    from mia_gb300 import synth
    lv, mov, ref = _level(size, 4.0, "ssd")
    o = O.Level(size, rate=4.0, cost="ssd", penalty_weight=1.0)
    o.set_images(mov, ref)
    # smooth: what varies over a tile grows with the amplitude, up to past
    # the ring's 10 planes, 16 rows and 64 columns
    p = synth.smooth_params(lv.csize, amplitude, seed=9)
    wo, co = o.warp(p), o.evaluate(p)[0]
    first = None
    for tz in (4, 8, 12, 16, 20, 24, 32):
        lv.set_path("split", (32, 8, tz))
        w = lv.warp(p)
        assert np.max(np.abs(w - wo)) <= 1e-5 * np.max(np.abs(mov)), tz
        # a voxel's sample does not depend on the tile that holds it
        first = w if first is None else first
        np.testing.assert_array_equal(w, first)
        assert abs(lv.evaluate(p)[0] - co) <= 1e-5 * co, tz


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e30, -3e6])
def test_displacements_that_are_not_numbers(value):
    """the device entry point takes parameters as they are: a coefficient
    that is not a usable number affects its voxels only, and the split path
    gives the plain path's image cost"""
    import torch
    size = (70, 20, 24)
    lv, mov, ref = _level(size, 6.0, "ssd")
    p = np.random.default_rng(3).normal(0.0, 1.0, lv.nparams)
    # in the middle of the grid, the z component
    c = [n // 2 for n in lv.csize]
    p[((c[2] * lv.csize[1] + c[1]) * lv.csize[0] + c[0]) * 3 + 2] = value
    d_p = torch.from_numpy(p).cuda()
    d_g = torch.empty(lv.nparams, dtype=torch.float64, device="cuda")
    d_c = torch.empty(2, dtype=torch.float64, device="cuda")
    cost = []
    for path in ("plain", "split"):
        lv.set_path(path)
        torch.cuda.synchronize()
        lv.evaluate_device(d_p.data_ptr(), d_g.data_ptr(), d_c.data_ptr())
        lv.sync()
        cost.append(d_c.cpu().numpy()[0])
    assert np.isfinite(cost[0])
    assert abs(cost[1] - cost[0]) <= 1e-5 * cost[0]


@pytest.mark.parametrize("hole", ["all", "one"])
def test_a_moving_image_that_is_not_a_number(hole):
    """the device entry point takes images as they are: voxels without a
    value are sampled as the lower bound of the clamp (at most 0), in the
    ring as in the plain path, also where the image has no value at all"""
    import torch

    import mia_gb300 as M
    from mia_gb300 import synth
    size = (70, 20, 24)
    rng = np.random.default_rng(8)
    mov, ref = rng.uniform(1.0, 2.0, (2, *size[::-1])).astype(np.float32)
    if hole == "all":
        mov[:] = np.nan
    else:
        mov[7, 9, 30] = np.nan
    d_mov, d_ref = torch.from_numpy(mov).cuda(), torch.from_numpy(ref).cuda()
    lv = M.Level(size, rate=6.0, cost="ssd")
    torch.cuda.synchronize()
    lv.set_images_device(d_mov.data_ptr(), d_ref.data_ptr())
    p = synth.smooth_params(lv.csize, 1.0, seed=2)
    warped, cost = [], []
    for path in ("plain", "split"):
        lv.set_path(path)
        cost.append(lv.evaluate(p)[0])
        warped.append(lv.warp(p))
    assert np.isfinite(cost[0]) and abs(cost[1] - cost[0]) <= 1e-5 * cost[0]
    np.testing.assert_array_equal(warped[1], warped[0])
    if hole == "all":
        assert np.all(warped[1] == 0.0)


@pytest.mark.parametrize("size", [(40, 24, 20), (70, 33, 21), (36, 41, 50)])
def test_batch_and_single_sums_of_tiles_outside_the_ring(size):
    """Images whose last x tile is narrow: its box leaves the padded copy, so
    its planes are sampled after the walk, and a batch adds their squares
    rounded, a single evaluation does not.  Over one minimizer step from the
    same start both take the same step (an SSD force does not depend on the
    sum), so the parameters have the same bits; each sum is off by at most 16
    additions per thread and 5 tree levels of 2^-24 relative (all terms are
    positive), so the costs differ by at most 2 * 22 * 2^-24."""
    from mia_gb300 import registration as R
    from mia_gb300 import synth
    ref = synth.blob_phantom(size[::-1], 8, sigma=(3.0, 6.0), seed=6)
    mov = np.roll(ref, 1, axis=2).astype(np.float32)
    mz = R.minimizer("gsl", maxiter=1, step=0.1)
    kw = dict(cost="ssd", penalty_weight=1.0)
    one = R.register_pair(mov, ref, 6.0, 1, mz, path="split", **kw)
    both = R.register_batch([(mov, ref), (mov, ref)], 6.0, 1, mz, **kw)
    for b in both:
        np.testing.assert_array_equal(b[0], one[0])
        assert b[3] == one[3] and abs(b[2] - one[2]) <= 44 * 2.0 ** -24 * abs(one[2])
