"""Grids so fine that a tile's shared memory does not fit a block: the split
path's launch is refused, the call reports it, writes nothing to the caller's
buffers and has nothing queued that still reads or writes them; the level's
other calls and the split path on an ordinary grid give what they always
give.

In a process of its own: a size that was refused must not count as raised for
the same kernel's later launches, and other tests raise it too.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import sys
import numpy as np
import mia_gb300 as M
from mia_gb300 import _lib, synth
from oracle import oracle as O

size, csize, tile, cost = eval(sys.argv[1])
ref = synth.blob_phantom(size[::-1], 6, sigma=(3.0, 8.0), seed=2)
mov = np.roll(ref, 1, axis=-1).astype(np.float32)
lv = M.Level(size, csize=csize, cost=cost)
lv.set_images(mov, ref)
p = synth.smooth_params(csize, 0.8, seed=4)
force = np.random.default_rng(1).normal(size=mov.shape + (len(size),)).astype(np.float32)


def others():   # what the level can do (a 3D level refuses a path's choice while its tile does not fit)
    if len(size) == 3:
        return [lv.translate(force)]
    lv.set_path("plain")
    r = [lv.translate(force), *lv.evaluate(p)]
    lv.set_path("split", tile)
    return r


want = others()
for k in range(20):
    q, grad = p.copy(), np.full(lv.nparams, 7.0)   # freed as soon as the call has failed
    if k % 2:
        q[k] = np.nan
    try:
        lv.evaluate_total(q, grad_out=grad)
    except _lib.MgrError as e:
        assert e.status == _lib.MGR_ERR_CUDA, e
    else:
        raise SystemExit("the launch was not refused")
    assert np.all(grad == 7.0)
    for f in (lv.value, lv.evaluate):
        try:
            f(q)
        except _lib.MgrError as e:
            assert e.status in (_lib.MGR_ERR_CUDA, _lib.MGR_ERR_ARG), e
        else:
            raise SystemExit("the launch was not refused")
    del q, grad
for x, y in zip(others(), want):
    np.testing.assert_array_equal(x, y)
# an ordinary grid on the same level and tile
g = tuple(n // 4 + 3 for n in size)
lv.set_grid(g)
lv.set_path("split", tile)
o = O.Level(size, csize=g, cost=cost, precision=O.PREC_F64)
o.set_images(mov, ref)
p = synth.smooth_params(g, 0.8, seed=5)
a, b = lv.evaluate(p), o.evaluate(p)
assert abs(a[0] - b[0]) <= 1e-5 * abs(b[0])
assert np.linalg.norm(a[2] - b[2]) <= 1e-4 * np.linalg.norm(b[2])
print("as expected")
"""


@pytest.mark.parametrize("case", [((33, 14, 49), (59, 32, 86), (32, 8, 4), "ncc"),
                                  ((33, 14, 49), (59, 32, 86), (32, 8, 4), "ssd"),
                                  ((64, 40), (390, 220), (64, 16), "ssd"),
                                  ((64, 40), (390, 220), (64, 16), "ncc")], ids=["3d-ncc", "3d-ssd", "2d-ssd", "2d-ncc"])
def test_a_refused_launch_touches_nothing(case):
    r = subprocess.run([sys.executable, "-c", SCRIPT, repr(case)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and "as expected" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
