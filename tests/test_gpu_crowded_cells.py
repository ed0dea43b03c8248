"""Push times of grids that are sparse but for a few full cells (a beam spot): a
cell far fuller than its neighbours gets whole warps.  The bounds are what a push
with a warp a cell took on a B200 (256 x 256 cells, 2 ions a cell and one cell of
8,000 / 40,000: 117 / 425 us), with a sixth more for the clock.  Four lanes a
cell, which the mean alone would choose, take 412 / 1,974 us.  Values are checked in
test_gpu_cells.py.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crowd,limit_us", [(8000, 137.0), (40000, 496.0)])
def test_one_full_cell_in_a_sparse_grid(crowd, limit_us):
    import pic_b200 as P
    from test_gpu_particles import lib_dx, make_pic, small_workload
    w = small_workload(256, 256, 2)
    dx, dy = lib_dx(w)
    rng = np.random.default_rng(crowd)
    cell = np.concatenate([np.repeat(np.arange(w.nx * w.ny), 2), np.full(crowd, 85 * w.nx + 128)])
    pts = np.zeros(len(cell), P.POINT_DTYPE)
    pts["x"] = (cell % w.nx + rng.random(len(cell))) * dx
    pts["y"] = (cell // w.nx + rng.random(len(cell))) * dy
    for k in ("vx", "vy", "vz"):
        pts[k] = rng.normal(0.0, 250.0, len(cell))
    ms, calls = (ctypes.c_double * 16)(), (ctypes.c_int64 * 16)()
    with make_pic(w) as pic:
        pic.set_phi(np.zeros(pic.nodes))
        pic.update_fields()
        pic.import_points(1, pts)
        pic.move_particles(1)
        P._check(P.lib().pic_set_profiling(pic.h, 1))
        us = []
        for _ in range(9):
            P._check(P.lib().pic_profile_read(pic.h, ms, calls, 1))
            pic.move_particles(1)
            pic.synchronize()
            P._check(P.lib().pic_profile_read(pic.h, ms, calls, 1))
            us.append(1e3 * (ms[0] + ms[1]))  # the push and the side list's kernel
        assert int(pic.bin_counts(1).max()) > 0.9 * crowd
    assert np.median(us) <= limit_us, us
