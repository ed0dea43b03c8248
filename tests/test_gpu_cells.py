"""The cell kernels' variants against the oracle: 4, 8 and 16 lanes a cell
(chosen by the particles a cell), uniform and varying Bz, with and without the
energy mesh, rows that a tile does not divide, empty cells, and cells far
fuller than the rest (several flushes of a lane's sums).

One push from identical particles, then the deposit of the new positions.
Tolerances, each from the arithmetic:
  * final_mesh: a particle's position is off by at most 2e-6 cell (the bound
    the push is held to), which moves at most that share of its weight between
    nodes: 2 axes x 2e-6, plus the 20-bit axis weights' 2 x 2^-21 -> 6e-6 of
    the fullest node;
  * energy mesh: velocities to 2e-5 v_th, so energies to about 6e-5 of the
    thermal one, averaged over the cell's particles; 1e-4 of the fullest node;
  * total charge: the particles' weights sum exactly, 1e-12;
  * a second push of the same state: the same bits (integer sums).
"""
import numpy as np
import pytest

from test_gpu_particles import lib_dx, make_pic, oracle_grid, oracle_species, small_workload

pytestmark = pytest.mark.gpu


def _points(w, s, ppc, crowd, seed):
    import pic_configs as C
    import pic_b200 as P
    pts = C.host_points(w, s, seed, ppc=ppc)
    dx, dy = lib_dx(w)
    # some cells empty
    cell = np.floor(pts["y"] / dy).astype(int) * w.nx + np.floor(pts["x"] / dx).astype(int)
    pts = pts[cell % 7 != 3]
    # and two crowded ones, one of them in the last column and row
    rng = np.random.default_rng(seed)
    extra = []
    for gx, gy, n in ((w.nx // 2, 1, crowd), (w.nx - 1, w.ny - 1, crowd // 3)):
        e = np.zeros(n, P.POINT_DTYPE)
        e["x"], e["y"] = (gx + rng.random(n)) * dx, (gy + rng.random(n)) * dy
        sig = np.std(pts["vx"])
        for k in ("vx", "vy", "vz"):
            e[k] = rng.normal(0, sig, n)
        extra.append(e)
    return np.concatenate([pts] + extra)


@pytest.mark.parametrize("ppc,crowd", [(1, 9000), (5, 20000), (20, 300), (20, 40000), (70, 9000)])
@pytest.mark.parametrize("nx,ny,profile,energy", [(37, 29, False, True), (65, 40, True, True), (130, 5, False, False),
                                                  (33, 31, True, False)])
def test_push_and_deposit_of_every_variant(oracle, ppc, crowd, nx, ny, profile, energy):
    w = small_workload(nx, ny, max(ppc, 1))
    w.b0 = 0.015
    dx, dy = lib_dx(w)
    rng = np.random.default_rng(nx * 100 + ppc)
    phi = rng.normal(0, 5.0, w.GX * w.GY)
    bz = 0.01 + 0.01 * rng.random(w.GX * w.GY) if profile else np.full(w.GX * w.GY, w.b0)
    oracle.overwrite_phi(w.GX, w.GY, oracle.Electrodes(w.rects), phi)
    ef = oracle.efield(w.GX, w.GY, dx, dy, phi)
    g = oracle_grid(oracle, w)
    meshes = []
    for _ in range(2):
        with make_pic(w, deposit_energy=energy) as pic:
            if profile:
                pic.set_bz(bz)
            pic.set_phi(phi)
            pic.update_fields()
            got = []
            for s in range(2):
                pts = _points(w, s, ppc, crowd, 5 + s)
                pic.import_points(s, pts)
                pic.move_particles(s)
                pic.zero_rho()
                pic.charge_deposition(s)
                got.append((pts, pic.final_mesh(s), pic.energy_mesh(s), pic.count(s)))
            meshes.append(got)
    for s in range(2):
        pts, final, en, count = meshes[0][s]
        assert np.array_equal(final, meshes[1][s][1]) and np.array_equal(en, meshes[1][s][2])
        ref = pts.copy()
        oracle.push(g, ref, w.species[s][0] / w.species[s][1], w.dt, ef, bz)
        live = ref[ref["pointer"] != -1]
        assert abs(count - len(live)) <= 3  # within rounding of a wall
        sp, weigh = oracle_species(oracle, w, s)
        rho = np.zeros(g.nodes)
        final_o, en_o = oracle.deposit(g, live, sp, weigh, 8.854e-12, rho)
        unit = weigh * dx * dy  # one particle
        slack = abs(count - len(live)) * unit
        assert np.abs(final - final_o).max() <= 6e-6 * final_o.max() + slack
        assert abs(final.sum() - count * unit) <= 1e-12 * final.sum()
        if energy:
            assert np.abs(en - en_o).max() <= 1e-4 * en_o.max() + slack * en_o.max() / unit
        else:
            assert not en.any()
