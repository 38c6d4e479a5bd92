"""The 2D penalty's cells packed with the level's other tables (small grids)
and uploaded from the shared table (from 256 KB on, about 13000 cells): just
below and above, on levels whose grid moves from one to the other and back,
the values and gradients of fresh levels and of the oracle (the parity tests'
tolerances, 1e-5 and 1e-4)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grids", [[(16, 16), (20, 19), (16, 16)], [(40, 30), (5, 5), (41, 30)]])
def test_grids_on_both_sides(grids):
    import mia_gb300 as M
    from mia_gb300 import synth
    from oracle import oracle as O
    size = (120, 90)
    ref = synth.blob_phantom(size[::-1], 8, sigma=(3.0, 8.0), seed=4)
    mov = np.roll(ref, 2, axis=1).astype(np.float32)
    kw = dict(cost="ssd", penalty_weight=3.0, div=1.5, curl=0.5)
    lv = M.Level(size, csize=grids[0], **kw)
    lv.set_images(mov, ref)
    for g in grids:
        lv.set_grid(g)
        for tile in [(32, 16), (64, 8)]:   # a new tile keeps the cells
            lv.set_path("split", tile)
            p = synth.smooth_params(g, 1.2, seed=g[0])
            got = lv.evaluate(p)
            fresh = M.Level(size, csize=g, **kw)
            fresh.set_images(mov, ref)
            fresh.set_path("split", tile)
            for x, y in zip(got, fresh.evaluate(p)):
                np.testing.assert_array_equal(x, y)
            fresh.close()
        o = O.Level(size, csize=g, precision=O.PREC_F64, **kw)
        o.set_images(mov, ref)
        _, op, _, ogp = o.evaluate(p)
        assert abs(got[1] - op) <= 1e-5 * abs(op)
        assert np.linalg.norm(got[3] - ogp) <= 1e-4 * np.linalg.norm(ogp)
        assert abs(lv.value(p)[1] - op) <= 1e-5 * abs(op)
    lv.close()
