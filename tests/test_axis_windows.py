"""The per-coefficient voxel ranges that the 2D adjoint kernel sums over (CPU).

For every coefficient of a tile's slot the kernel (mia_gb300/csrc/split.cu,
adjoint2_body) takes the tile's voxels i in the coefficient's range and reads
the weight at i * 4 + (o - start[i]).  The ranges hold exactly the voxels
whose window start .. start + 3 contains the coefficient, so that the index
stays inside the voxel's four weights, on grids of any spacing: coarser than
the voxels, one to one, and so fine that windows leave coefficients out.
"""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

_ip = ctypes.POINTER(ctypes.c_int)
_fp = ctypes.POINTER(ctypes.c_float)


@pytest.fixture(scope="module")
def shim():
    d = tempfile.mkdtemp(prefix="mgr_axis_")
    so = os.path.join(d, "libaxisshim.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-ffp-contract=off", "-shared", "-o", so,
                           os.path.join(HERE, "axis_tables_shim.cc"),
                           os.path.join(ROOT, "mia_gb300", "csrc", "tables.cc")])
    L = ctypes.CDLL(so)
    L.shim_axis.argtypes = [ctypes.c_int] * 3 + [_ip, _fp, _ip, _ip]

    def axis(n, nc, tile):
        a = [np.zeros(n, np.int32), np.zeros((n, 4), np.float32), np.zeros((nc, 2), np.int32), np.zeros(n, np.int32)]
        ac = L.shim_axis(n, nc, tile, *(x.ctypes.data_as(_fp if x.dtype == np.float32 else _ip) for x in a))
        return (ac, *a)
    return axis


SIZES = [2, 3, 7, 8, 9, 16, 31, 33, 64, 65, 200]


def grids(n):
    return sorted({4, 5, 6, 9, n // 8 + 4, n // 2 + 3, n, n + 2, n + 3, 2 * n + 2, 3 * n, 4 * n, 5 * n, 6 * n + 1,
                   9 * n + 3} - set(range(4)))


@pytest.mark.parametrize("n", SIZES)
def test_a_range_is_the_voxels_whose_window_holds_the_coefficient(shim, n):
    for nc in grids(n):
        _, start, weight, win, _ = shim(n, nc, 16)
        assert np.all(np.diff(start) >= 0)
        for o in range(nc):
            lo, hi = win[o]
            held = np.flatnonzero((start <= o) & (o <= start + 3))
            assert 0 <= lo <= hi <= n
            np.testing.assert_array_equal(np.arange(lo, hi), held, err_msg="nc %d coefficient %d" % (nc, o))


@pytest.mark.parametrize("tile", [8, 16, 32, 64])
@pytest.mark.parametrize("n", SIZES)
def test_a_tile_sums_each_weight_once(shim, n, tile):
    """the kernel's loop over a tile's slot in whole numbers: each voxel's
    four weights are met once each where the coefficient is in the grid"""
    for nc in grids(n):
        ac, start, _, win, atile0 = shim(n, nc, tile)
        for b in range((n + tile - 1) // tile):
            v0, e = b * tile, min(tile, n - b * tile)
            met = np.zeros((e, 4), int)
            for o in range(ac):
                c = atile0[b] + o
                lo, hi = win[c] if c < nc else (0, 0)
                for i in range(max(lo - v0, 0), min(hi - v0, e)):
                    k = o - (start[v0 + i] - atile0[b])
                    assert 0 <= k <= 3, (nc, b, o, i)
                    met[i, k] += 1
            inside = start[v0:v0 + e, None] + np.arange(4)[None, :] < nc
            np.testing.assert_array_equal(met, inside.astype(int))
