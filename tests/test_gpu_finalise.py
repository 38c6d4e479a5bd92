"""The reductions at the end of an evaluation where their batches end (tiles
and gather blocks below, at and above the threads that add them), and the
kernels that finalise a cost against one another.

Tolerances: the parity tests' own, costs 1e-5 relative and gradients 1e-4
relative L2 against the all-double oracle.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _level(size, rate, cost):
    import mia_gb300 as M
    from mia_gb300 import synth
    kw = dict(rate=rate, cost=cost, penalty_weight=2.0, curl=0.5)
    lv = M.Level(size, **kw)
    ref = synth.blob_phantom(size[::-1], 8, sigma=(2.0, 5.0), seed=3)
    mov = (np.roll(ref, 1, axis=1) * 1.1).astype(np.float32)
    lv.set_images(mov, ref)
    return lv, mov, ref, synth.smooth_params(lv.csize, 1.0, seed=7), kw


# gather blocks of 32 coefficients: 2, 32 and 33 rows of them, and more than
# the 1024 that one batch of the last block's loads covers
@pytest.mark.parametrize("cost", ["ssd", "ncc"])
@pytest.mark.parametrize("size,rate", [((9, 7), 2.0), ((64, 61), 2.0), ((380, 372), 2.0), ((12, 10, 9), 4.0),
                                       ((66, 64, 62), 2.0)])
def test_sums_over_tiles_and_blocks(size, rate, cost):
    from oracle import oracle as O
    lv, mov, ref, p, kw = _level(size, rate, cost)
    o = O.Level(size, precision=O.PREC_F64, **kw)
    o.set_images(mov, ref)
    oi, op, ogi, ogp = o.evaluate(p)
    ov = o.value(p)
    ci, cp, gi, gp, gt = lv.evaluate(p)
    assert abs(ci - oi) <= 1e-5 * abs(oi) and abs(cp - op) <= 1e-5 * abs(op)
    assert np.linalg.norm(gi - ogi) <= 1e-4 * np.linalg.norm(ogi)
    assert np.linalg.norm(gp - ogp) <= 1e-4 * np.linalg.norm(ogp)
    vi, vp = lv.value(p)
    assert abs(vi - ov[0]) <= 1e-5 * abs(ov[0]) and abs(vp - ov[1]) <= 1e-5 * abs(ov[1])


@pytest.mark.parametrize("cost", ["ssd", "ncc"])
@pytest.mark.parametrize("size", [(70, 41), (300, 290), (40, 20, 17), (130, 90, 33)])
def test_the_cost_does_not_depend_on_who_finalises_it(size, cost):
    """evaluate (the gather, for SSD) and force (the warp kernel or the one
    after it): the same tile sums in the same order, the same bits"""
    lv, _, _, p, _ = _level(size, 8.0, cost)
    ci = lv.evaluate(p)[0]
    fc = lv.force(p)[0]
    assert fc == ci
    if cost == "ssd":
        assert lv.value(p)[0] == ci


@pytest.mark.parametrize("cost", ["ssd", "ncc"])
@pytest.mark.parametrize("size", [(70, 41), (40, 20, 17)])
def test_value_from_host_memory(size, cost, monkeypatch):
    """parameters and costs in the caller's host memory or copied: the same
    bits; non-finite parameters are refused, the level stays usable"""
    import mia_gb300 as M
    from mia_gb300 import _lib
    lv, mov, ref, p, kw = _level(size, 8.0, cost)
    monkeypatch.setenv("MGR_HOST_COPY", "1")
    staged = M.Level(size, **kw)
    monkeypatch.delenv("MGR_HOST_COPY")
    staged.set_images(mov, ref)
    want = staged.value(p)
    assert lv.value(p) == want
    for bad in (np.nan, np.inf):
        q = p.copy()
        q[-1] = bad
        for level in (lv, staged):
            with pytest.raises(_lib.MgrError):
                level.value(q)
            assert level.value(p) == want
    assert lv.evaluate(p)[:2] == staged.evaluate(p)[:2]
