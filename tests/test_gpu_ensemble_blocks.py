"""The batched solve's block shapes: ensembles below and above the node count from
which its blocks take half an SM each, of instances at the edges of tiles (one
tile, a node more or less than a multiple of the 32-node core, long and narrow,
periodic in y, levels smaller than a tile, no level above the fused ones), with
one block and with many an instance.

Each instance's potential after a step is compared with that of a context of its
own stepped on the same particles (the charge is the same, whole numbers).  Both
solve to a relative residual of 1e-10, with different preconditioners, so each is
off by at most the condition number times that: below 4 (n / pi)^2 = 1.7e4 for
the n <= 205 cells of the widest grid here, 1.7e-6 each; 4e-6 of |phi| in the
2-norm is asserted.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _config(nx, ny, periodic, left):
    import pic_b200 as P
    import pic_configs as C
    rects = C.periodic_rects(nx, ny, left=left) if periodic else C.wall_rects(nx, ny, left=left)
    return P.make_config(nx, ny, nx * 2.5e-4, ny * 2.5e-4, 5e-11, C._species(nx, ny, 2, 1e15), rects,
                         warm=P.WARM_ZERO, tol=1e-10, periodic_y=periodic)


EDGES = [(4, 4, False), (31, 30, False), (62, 63, False), (64, 65, False), (95, 33, False), (40, 200, False),
         (64, 64, True), (70, 48, True), (160, 97, False)]


@pytest.mark.parametrize("sizes,half", [
    (EDGES, False),
    ([(200, 201, False)], False),
    (EDGES + [(190 + k % 16, 188 + k % 13, False) for k in range(42)], True),
])
def test_instances_match_single_contexts(sizes, half):
    import pic_b200 as P
    cfgs = [_config(nx, ny, per, 20.0 + k) for k, (nx, ny, per) in enumerate(sizes)]
    with P.Ensemble(cfgs) as E:
        assert (E.info()["solver_blocks"] > 200) == half
        for k in range(len(sizes)):
            for s in range(2):
                E[k].load_plasma(s, 2, 2.0, 3 * k + s)
        E.step(0)
        got = [(E[k].poisson_stats()[:2], E[k].phi(), E[k].rho()) for k in range(len(sizes))]
    for k in list(range(min(len(sizes), len(EDGES)))) + [len(sizes) - 1]:
        with P.Pic(cfgs[k]) as pic:
            for s in range(2):
                pic.load_plasma(s, 2, 2.0, 3 * k + s)
            pic.step(0)
            (it, rel), phi, rho = got[k]
            assert rel <= 1e-10 and 0 < it < 60
            assert np.array_equal(rho, pic.rho())
            d = np.linalg.norm(phi - pic.phi())
            assert d <= 4e-6 * np.linalg.norm(pic.phi()), (sizes[k], d)
