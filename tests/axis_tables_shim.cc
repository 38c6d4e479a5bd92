// C entry point over the product's per-axis table builder
// (mia_gb300/csrc/tables.cc), compiled by tests/test_axis_windows.py together
// with tables.cc so that the CPU tests can look at the tables without a GPU.
#include <algorithm>

#include "../mia_gb300/csrc/tables.hh"

// the adjoint starts (n), weights (n x 4), windows (nc x 2), the tiles' first
// coefficients (number of tiles, at most n) and the slot length (returned)
extern "C" int shim_axis(int n, int nc, int tile, int *as, float *aw, int *win, int *atile0)
{
    mgr::AxisHost h;
    mgr::build_axis(h, n, nc, tile);
    std::copy(h.as.begin(), h.as.end(), as);
    std::copy(h.aw.begin(), h.aw.end(), aw);
    std::copy(h.win.begin(), h.win.end(), win);
    std::copy(h.atile0.begin(), h.atile0.end(), atile0);
    return h.ac;
}
