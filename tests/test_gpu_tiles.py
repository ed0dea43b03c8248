"""The V-cycle's tile kernels at the sizes where their tiles end: grids a node
below, at and above a multiple of the 32-node core, one tile, one node more than
a tile, long and narrow ones, levels smaller than a tile, walled and periodic in
y.  Against the V-cycle with a kernel a half sweep: the same bits (each node's
arithmetic is the same), the right-hand side with large and tiny values mixed,
so that a halo node that is off by a rounding shows.
"""
import numpy as np
import pytest

from test_gpu_vcycle import run, vcycle_pic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,periodic,inner", [
    (62, 62, False, False), (63, 64, False, True), (64, 65, False, False), (95, 96, False, True),
    (97, 94, False, False), (500, 34, False, False), (34, 500, False, False), (40, 36, False, True),
    (64, 64, True, False), (33, 68, True, False), (70, 32, True, True), (300, 256, True, True),
    (1000, 60, False, True), (771, 389, False, True),
])
def test_tiles_match_per_sweep(nx, ny, periodic, inner):
    rng = np.random.default_rng(7 * nx + ny)
    with vcycle_pic(nx, ny, periodic, inner) as pic:
        rhs = (rng.standard_normal(pic.nodes) * 10.0 ** rng.integers(-6, 7, pic.nodes)).astype(np.float32)
        a = run(pic, rhs, 0)
        b = run(pic, rhs, 1)
    assert np.abs(a).max() > 0
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), \
        f"{np.count_nonzero(a != b)} nodes differ, max {np.abs(a - b).max():.3e}"
