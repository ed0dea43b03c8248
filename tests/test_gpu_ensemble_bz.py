"""Ensembles whose instances differ in the kind of their Bz, uniform or a profile:
each instance's step is the one it has beside instances of its own kind, bit for
bit (the charge and the energies are whole-number sums, the solve's sums are
ordered by the instance's size, and its particles are pushed with its own Bz's
arithmetic), also when an instance changes its kind between two steps, with and
without the captured step, and a run repeats bit for bit.
"""
import numpy as np
import pytest

from test_gpu_particles import export_state

pytestmark = pytest.mark.gpu

SIZES = [(40, 33), (65, 40), (33, 64), (48, 48)]
B0 = [0.013, 0.007, 0.019, 0.011]


def _configs():
    import pic_b200 as P
    import pic_configs as C
    return [P.make_config(nx, ny, nx * 2.5e-4, ny * 2.5e-4, 5e-11, C._species(nx, ny, 10, 1e15),
                          C.wall_rects(nx, ny, left=30.0 + k), b0=B0[k]) for k, (nx, ny) in enumerate(SIZES)]


def _profile(k):
    nx, ny = SIZES[k]
    return np.tile(0.004 + 0.016 * np.linspace(0, 1, nx + 1), ny + 1)


def _uniform(k):
    nx, ny = SIZES[k]
    return np.full((nx + 1) * (ny + 1), B0[k])


def _states(E):
    out = []
    for k in range(len(SIZES)):
        st = [E[k].phi()]
        for s in range(2):
            st += [E[k].final_mesh(s), E[k].energy_mesh(s)]
            e = export_state(E[k], s)
            a = np.stack([e[q].astype(np.float64) for q in ("cell", "fx", "fy", "vx", "vy", "vz")])
            st.append(a[:, np.lexsort(a)])
        out.append(st)
    return out


def _run(plan, graph=True):
    """plan: for each step, the instances whose Bz is a profile."""
    import pic_b200 as P
    with P.Ensemble(_configs()) as E:
        E.use_graph(graph)
        for k in range(len(SIZES)):
            for s in range(2):
                E[k].load_plasma(s, 10, (2.0, 0.026)[s], 5 * k + s)
        now = set()
        for it, want in enumerate(plan):
            for k in now ^ set(want):
                E[k].set_bz(_profile(k) if k in want else _uniform(k))
            now = set(want)
            E.step(it)
        return _states(E)


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("graph", [True, False])
def test_instances_do_not_depend_on_the_others_bz(graph):
    uniform = _run([()] * 4, graph)
    profile = _run([(0, 1, 2, 3)] * 4, graph)
    for mixed in ((2,), (0, 3), (0, 1, 2)):
        got = _run([mixed] * 4, graph)
        for k in range(len(SIZES)):
            assert _same(got[k], (profile if k in mixed else uniform)[k]), (mixed, k)


def test_bz_kind_changes_between_steps():
    uniform = _run([()] * 5)
    plan = [(), (1,), (1, 3), (), (3,)]
    a, b = _run(plan), _run(plan)
    alone = {k: _run([(0, 1, 2, 3) if k in p else () for p in plan])[k] for k in (1, 3)}
    for k in range(len(SIZES)):
        assert _same(a[k], b[k])
    assert _same(a[0], uniform[0]) and _same(a[2], uniform[2])
    for k in (1, 3):
        assert _same(a[k], alone[k])
