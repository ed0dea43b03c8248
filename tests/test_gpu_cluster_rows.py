"""Which grids the one-cluster Poisson solve takes, and its halo rows: periodic in
y with fewer rows on a distributed level than the halo has (halo rows would be
images two periods away: such grids go to the kernels), periodic with two
distributed levels, bands of no row and of very many, levels one node below and
above the size from which they are distributed.

The solver that ran is told by the launches of a solve: the cluster's is one
launch, the kernels' are several.  Both are PCG with the same V-cycle, node for
node, and the same alpha and beta, so iterations and potentials are equal to the
last bit.
"""
import ctypes

import numpy as np
import pytest

from test_gpu_cluster_solve import _pic

pytestmark = pytest.mark.gpu


def _solve(pic, k, rho):
    import pic_b200 as P
    n0, n1 = ctypes.c_int64(0), ctypes.c_int64(0)
    pic.set_rho(rho)
    P.lib().pic_launch_count(pic.h, ctypes.byref(n0))
    pic.poisson_solve(k)
    P.lib().pic_launch_count(pic.h, ctypes.byref(n1))
    return n1.value - n0.value, pic.poisson_stats()[:2], pic.phi(), pic.rho()


@pytest.mark.parametrize("nx,ny,periodic,inner,cluster", [
    # distributed levels of fewer rows than the halo: 4 rows on level 0, 4 on level 1
    (375, 4, True, False, False), (400, 4, True, False, False), (1000, 4, True, False, False),
    (1198, 4, True, False, False), (749, 8, True, False, False), (760, 8, True, False, False),
    (798, 8, True, False, False),
    # one node column less: that level is kept whole by every block
    (374, 4, True, False, True), (748, 8, True, False, True),
    # periodic, two distributed levels
    (100, 96, True, False, True), (60, 192, True, True, True), (180, 64, True, True, True), (90, 144, True, False, True),
    # walls: long and narrow (bands of no row; of 1,000 columns the halos do not fit the
    # shared memory), too many rows, the largest and one too large
    (300, 12, False, False, True), (600, 12, False, False, True), (1000, 12, False, False, False),
    (14, 900, False, False, False), (500, 16, False, True, True),
    # the most rows, and one more
    (20, 640, False, False, True), (20, 641, False, False, False), (19, 640, True, False, True), (7, 1600, True, False, False),
    (117, 117, False, True, True), (118, 118, False, True, False),
])
def test_solver_and_halo_rows(nx, ny, periodic, inner, cluster):
    import pic_b200 as P
    rng = np.random.default_rng(nx * 1000 + ny)
    rhos = None
    with _pic(nx, ny, periodic, inner, P.WARM_PREVIOUS) as pic:
        rhos = [rng.normal(0.0, 1e6, pic.nodes) for _ in range(2)]
        res = []
        for graph in (1, 0):  # 1: the default
            assert P.lib().pic_set_poisson_graph(pic.h, graph) == 0
            pic.set_phi(np.zeros(pic.nodes))
            res.append([_solve(pic, k, rhos[k]) for k in range(2)])
    for a, b in zip(*res):
        assert (a[0] == 1) == cluster, a[0]
        assert b[0] > 1
        assert a[1][1] <= 1e-12
        assert a[1][0] == b[1][0]
        assert np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3])
