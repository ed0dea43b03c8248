"""The one-cluster Poisson solve (grids up to 14,000 nodes) against the
multi-kernel solve of the same system (pic_set_poisson_graph(0)): square, odd
and elongated grids, bands of few and of many rows, an inner electrode,
periodic in y, levels that are distributed and levels that every block keeps,
and grids too large for it.

Both are PCG with the same V-cycle, node for node, and alpha and beta are
summed in the same order, so iterations and potentials are equal to the last
bit.  |r0|^2 is not, and its rounding (a relative 2^-53 a term, summed) is
allowed 1e-6.  The field that the next push sees is the one that a fresh E field
of the same potential gives, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pic(nx, ny, periodic, inner, warm):
    import pic_b200 as P
    import pic_configs as C
    dx, dy = 2.5e-4, 2.0e-4
    box = (nx // 3, ny // 3, nx // 3 + max(1, nx // 8), ny // 3 + max(1, ny // 8), 75.0)
    if periodic:
        rects = C.periodic_rects(nx, ny, left=40.0, inner=box if inner else None)
    else:
        rects = C.wall_rects(nx, ny, left=40.0, top=-5.0) + ([box] if inner else [])
    cfg = P.make_config(nx, ny, nx * dx, ny * dy, 5e-11, C._species(nx, ny, 6, 1e15), rects, b0=0.01,
                        warm=warm, tol=1e-12, periodic_y=periodic)
    return P.Pic(cfg)


def _state(pic, s):
    from test_gpu_particles import export_state, multiset
    return multiset(export_state(pic, s))


@pytest.mark.parametrize("nx,ny,periodic,inner", [
    (4, 4, False, False), (20, 9, False, False), (32, 32, False, True), (33, 30, False, False),
    (40, 300, False, True), (300, 40, False, True), (57, 58, False, False), (64, 64, False, True),
    (101, 99, False, True), (128, 128, False, False), (150, 77, False, True), (210, 210, False, True),
    (48, 48, True, False), (90, 64, True, True), (200, 96, True, True), (60, 320, True, False),
    (7, 300, False, False), (1500, 20, False, False), (117, 117, False, True), (118, 118, False, True), (90, 150, True, False),
    (212, 212, False, False),
])
def test_cluster_solve_matches_the_kernels(nx, ny, periodic, inner):
    import pic_b200 as P
    rng = np.random.default_rng(nx * 1000 + ny)
    with _pic(nx, ny, periodic, inner, P.WARM_PREVIOUS) as pic:
        res = {}
        for graph in (1, 0):  # 1: the default, the cluster solve
            assert P.lib().pic_set_poisson_graph(pic.h, graph) == 0
            r = np.random.default_rng(nx * 1000 + ny)
            pic.set_phi(np.zeros(pic.nodes))
            out = []
            for k in range(2):  # the second from the first's potential
                rho = r.normal(0.0, 1e6, pic.nodes)
                pic.set_rho(rho)
                pic.poisson_solve(k)
                it, rel, _ = pic.poisson_stats()
                # (periodic in y with rows that do not halve twice: one level, hundreds of iterations)
                assert rel <= 1e-12 and 0 < it < (1000 if periodic and ny % 4 else 60)
                out.append((it, pic.phi(), pic.rho(), P.Pic.poisson_start_relres(pic)))
            res[graph] = out
        for a, b in zip(res[1], res[0]):
            assert a[0] == b[0]
            assert np.array_equal(a[2], b[2])                       # the right-hand side left in rho
            assert np.array_equal(a[1], b[1])
            assert abs(a[3] - b[3]) <= 1e-6 * b[3]
        # the field of the next push
        P.lib().pic_set_poisson_graph(pic.h, 1)
        phi = None
        states = []
        for fresh in (False, True):
            for s in range(2):
                pic.load_plasma(s, 6, 2.0, 9 + s)
            if not fresh:
                pic.set_phi(np.zeros(pic.nodes))
                pic.set_rho(rng.normal(0.0, 1e6, pic.nodes))
                pic.poisson_solve(5)
                phi = pic.phi()
            else:
                pic.set_phi(phi)
                pic.update_fields()
            for s in range(2):
                pic.move_particles(s)
            states.append([_state(pic, s) for s in range(2)])
        for s in range(2):
            assert np.array_equal(states[0][s], states[1][s])


def test_cluster_solve_iteration_limit():
    import pic_b200 as P
    with _pic(100, 80, False, True, P.WARM_ZERO) as pic:
        pic.set_poisson(warm=P.WARM_ZERO, tol=1e-12, maxit=2)
        rho = np.random.default_rng(1).normal(0.0, 1e6, pic.nodes)
        pic.set_rho(rho)
        with pytest.raises(P.PicError) as e:
            pic.poisson_solve(0)
        assert e.value.status == -4
        assert pic.poisson_stats()[0] == 2
        pic.set_poisson(warm=P.WARM_ZERO, tol=1e-10, maxit=100)
        pic.set_rho(rho)
        pic.poisson_solve(1)
        assert pic.poisson_stats()[1] <= 1e-10
