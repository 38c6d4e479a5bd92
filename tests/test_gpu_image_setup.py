"""The image set-up passes (coefficients, clamp bounds, mirror-padded copy,
means) at the sizes where their tiling can go wrong: lines shorter than the
halo, one below / at / above a block's 32 lines, lines long enough to lower
the lines per block.

A shift by whole voxels has a known answer: the image itself, its index
folded at the borders.  Shifts of up to 24 voxels read every part of the
padded copy and the folds behind it.

Tolerance.  Where a tap is wrong the error is of the size of the image.  The
rounding: the displacement is a sum of products with weights that add up to
1, at most 12 roundings of 2^-24 relative (three axes of four terms), the
sample point one more of its own size; so a point is off by at most
d = 12 * 2^-24 * |shift| + 2^-24 * (size + |shift|).  A cubic spline through
values of at most m has coefficients of at most 3^dim m and slopes of at most
that (its derivative's weights add up to at most 1 in magnitude per axis), so
the sample is off by at most dim * d * 3^dim m, and by 64 roundings of the
tap sum, 64 * 2^-24 * 3^dim m.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(2, 3, 4), (17, 16, 18), (31, 33, 32), (65, 2, 40), (40, 35, 5), (1030, 9, 3), (12, 700, 2), (9, 6, 640),
         (2, 2), (33, 31), (64, 15), (2050, 7), (10, 1100)]


def fold(i, n):
    i = np.abs(i) % (2 * n - 2)
    return np.where(i < n, i, 2 * n - 2 - i)


@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
def test_whole_voxel_shifts(size):
    import mia_gb300 as M
    dim = len(size)
    rng = np.random.default_rng(sum(size))
    # both signs, so that the clamp at 0 is not reached
    mov = rng.uniform(-1.0, 1.0, size[::-1]).astype(np.float32)
    lv = M.Level(size, csize=(5,) * dim, cost="ssd")
    lv.set_images(mov, mov)
    for shift in [(0, 0, 0), (1, -2, 3), (-16, 15, -14), (24, -21, 19)]:
        shift = shift[:dim]
        got = lv.warp(np.tile(np.array(shift, np.float64), lv.nparams // dim))
        idx = [fold(np.arange(n) - s, n) for n, s in zip(size, shift)]
        want = mov[np.ix_(*idx[::-1])]
        e = 2.0 ** -24
        d = 12 * e * max(map(abs, shift)) + e * (max(size) + max(map(abs, shift)))
        tol = 3.0 ** dim * (dim * d + 64 * e)
        assert tol < 0.1
        assert np.max(np.abs(got - want)) <= tol, shift
    lv.close()


@pytest.mark.parametrize("size", [(61, 47), (45, 38, 29), (7, 9, 300)])
def test_new_images_on_a_kept_level(size):
    """a second pair on the same level gives what a fresh level gives, and the
    device entry point what the host one gives, bit for bit; the costs and
    gradients (with the means, NCC's centres) those of the oracle"""
    import torch

    import mia_gb300 as M
    from oracle import oracle as O
    rng = np.random.default_rng(5)
    shape = size[::-1]
    a, b, c = (rng.normal(size=shape).astype(np.float32) for _ in range(3))
    d = (c + 0.2 * rng.normal(size=shape)).astype(np.float32)
    kw = dict(rate=6.0, cost="ncc", penalty_weight=2.0) if min(size) > 20 else dict(csize=(5, 5, 40), cost="ncc")
    lv = M.Level(size, **kw)
    p = rng.normal(0.0, 0.3, lv.nparams)
    lv.set_images(a, b)
    lv.evaluate(p)
    dc, dd = torch.from_numpy(c).cuda(), torch.from_numpy(d).cuda()
    torch.cuda.synchronize()
    lv.set_images_device(dc.data_ptr(), dd.data_ptr())
    got = lv.evaluate(p)
    fresh = M.Level(size, **kw)
    fresh.set_images(c, d)
    want = fresh.evaluate(p)
    for x, y in zip(got, want):
        np.testing.assert_array_equal(x, y)
    o = O.Level(size, precision=O.PREC_F64, **kw)
    o.set_images(c, d)
    assert abs(got[0] - o.evaluate(p)[0]) <= 1e-5 * abs(got[0])


# the recursion walks a line in batches of 8 values
@pytest.mark.parametrize("size", [(8, 9, 10), (11, 16, 17), (18, 19, 24), (25, 26, 27), (10, 9), (17, 18), (26, 33)],
                         ids=lambda s: "x".join(map(str, s)))
def test_line_lengths_about_the_batches(size):
    test_whole_voxel_shifts(size)
