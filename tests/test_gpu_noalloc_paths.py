"""The allocation-free deposit's two layouts (four words a cell up to 2^17 cells,
a word a node beyond) and its copies of the cell sums, at their edges: one cell,
one row, the largest grid of the one and the smallest of the other, the largest
the scratch takes, point counts around the copies' steps and around a warp and a
block, dead points and points outside, every point in one cell, none at all.
Against whole-number sums in numpy: the weights are exact products of 20-bit axis
weights, so the meshes are equal bit for bit.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 2.5e-4
EPS0 = 8.854187817e-12


def expected(x, y, alive, nx, ny, species, rho0):
    dx, dy = nx * DX / nx, ny * DX / ny
    sx, sy = x * (1.0 / dx), y * (1.0 / dy)
    ok = alive & (sx >= 0) & (sy >= 0) & (sx < nx) & (sy < ny)
    sx, sy = sx[ok], sy[ok]
    gx, gy = sx.astype(np.int64), sy.astype(np.int64)
    below = np.float32(1) - np.float32(2.0 ** -24)
    ax, ay = (np.rint(np.minimum((s - g).astype(np.float32), below).astype(np.float64) * 2 ** 20).astype(np.uint64)
              for s, g in ((sx, gx), (sy, gy)))
    one = np.uint64(1 << 20)
    sums = np.zeros((ny + 1) * (nx + 1), np.uint64)
    k = gy * (nx + 1) + gx
    for off, w in ((0, (one - ax) * (one - ay)), (1, ax * (one - ay)), (nx + 1, (one - ax) * ay), (nx + 2, ax * ay)):
        np.add.at(sums, k + off, w)
    xmax, ymax = nx * DX, ny * DX
    weighing = species.actual_count * (xmax * ymax) / (species.sim_count * dx * dy * dx * dy)
    final = sums.astype(np.float64) * (2.0 ** -40 * (dx * dy) * weighing)
    return final, rho0, -species.charge / EPS0


@pytest.mark.parametrize("nx,ny,n", [
    (1, 1, 1), (1, 1, 4097), (1, 500, 33), (500, 1, 70000), (7, 5, 0), (7, 5, 31), (7, 5, 257),
    (8, 8, 8191), (8, 8, 8192), (8, 8, 16384), (8, 8, 131072), (8, 8, 300001),
    (362, 362, 50001), (363, 361, 50001), (362, 363, 50001), (723, 723, 50001), (64, 64, 600000),
])
@pytest.mark.parametrize("one_cell", [False, True])
def test_deposit_matches_whole_number_sums(nx, ny, n, one_cell):
    import torch
    import pic_b200 as P
    rng = np.random.default_rng(nx * 7919 + ny * 31 + n)
    x = rng.uniform(-0.02, 1.02, n) * nx * DX
    y = rng.uniform(-0.02, 1.02, n) * ny * DX
    if one_cell:
        x, y = (rng.uniform(0, 1, n) + nx - 1) * DX, (rng.uniform(0, 1, n) + ny // 2) * DX
    alive = rng.random(n) > 0.05
    pts = torch.zeros(max(n, 1), 7, dtype=torch.float64)
    pts[:n, 0], pts[:n, 1] = torch.from_numpy(x), torch.from_numpy(y)
    pts.view(torch.int32)[:n, 12] = torch.from_numpy(np.where(alive, 5, -1).astype(np.int32))
    pts = pts.cuda()
    nodes = (nx + 1) * (ny + 1)
    rho0 = rng.normal(size=nodes)
    rho = torch.from_numpy(rho0.copy()).cuda()
    final = torch.full((nodes,), np.nan, dtype=torch.float64, device="cuda")
    sd = P.SpeciesDesc(-1.6e-19, 9.1e-31, float(max(n, 1)), 1e15)
    for _ in range(2):  # the scratch is used again
        rho.copy_(torch.from_numpy(rho0))
        P._check(P.lib().pic_deposit_points_noalloc(
            pts.data_ptr(), n, nx, ny, nx * DX, ny * DX, ctypes.byref(sd), 0.0, EPS0, final.data_ptr(),
            rho.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    want, r0, chrg = expected(x, y, alive, nx, ny, sd, rho0)
    got = final.cpu().numpy()
    assert np.array_equal(got, want)
    # rho += f * chrg, whose product may be fused: one rounding of it
    assert np.all(np.abs(rho.cpu().numpy() - (r0 + want * chrg)) <= 2.0 ** -52 * (np.abs(want * chrg) + np.abs(r0)))
