"""The allocation-free deposit of few points: on the largest grid whose cells fit
into the scratch it takes no longer than on one that is a column larger, where the
sums are kept by nodes (a tenth is allowed for timing), and both layouts give the
same sums at the count where they change over.  Values of both against
whole-number sums in test_gpu_noalloc_paths.py.
"""
import ctypes

import numpy as np
import pytest

from test_gpu_noalloc_paths import DX, EPS0, expected

pytestmark = pytest.mark.gpu


def _call(pts, n, nx, ny, sd, final, rho):
    import torch
    import pic_b200 as P
    P._check(P.lib().pic_deposit_points_noalloc(
        pts.data_ptr(), n, nx, ny, nx * DX, ny * DX, ctypes.byref(sd), 0.0, EPS0, final.data_ptr(),
        rho.data_ptr(), torch.cuda.current_stream().cuda_stream))


def _points(rng, n, nx, ny):
    import torch
    pts = torch.zeros(n, 7, dtype=torch.float64)
    pts[:, 0], pts[:, 1] = (torch.from_numpy(rng.random(n) * k * DX) for k in (nx, ny))
    return pts.cuda()


@pytest.mark.parametrize("n", [300, 3000, 30000])
def test_few_points_cost_no_more_by_cells(n):
    import torch
    import pic_b200 as P
    rng = np.random.default_rng(n)
    sd = P.SpeciesDesc(-1.6e-19, 9.1e-31, float(n), 1e15)
    graphs, keep = [], []
    for nx, ny in ((362, 362), (363, 362)):
        pts = _points(rng, n, nx, ny)
        final, rho = (torch.zeros((nx + 1) * (ny + 1), dtype=torch.float64, device="cuda") for _ in range(2))
        _call(pts, n, nx, ny, sd, final, rho)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(50):
                _call(pts, n, nx, ny, sd, final, rho)
        graphs.append(g)
        keep.append((pts, final, rho))
    ms = [[], []]
    for _ in range(15):
        for k, g in enumerate(graphs):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.replay()
            b.record()
            b.synchronize()
            ms[k].append(a.elapsed_time(b))
    small, large = np.median(ms[0]), np.median(ms[1])
    assert small <= 1.1 * large, (20 * small, 20 * large)


@pytest.mark.parametrize("nx,ny", [(20, 7), (64, 33), (362, 362)])
def test_sums_where_the_layout_changes(nx, ny):
    import torch
    import pic_b200 as P
    rng = np.random.default_rng(nx)
    for n in (3 * nx * ny - 1, 3 * nx * ny, 3 * nx * ny + 1):
        pts = _points(rng, n, nx, ny)
        sd = P.SpeciesDesc(-1.6e-19, 9.1e-31, float(n), 1e15)
        final, rho = (torch.zeros((nx + 1) * (ny + 1), dtype=torch.float64, device="cuda") for _ in range(2))
        _call(pts, n, nx, ny, sd, final, rho)
        p = pts.cpu().numpy()
        want, _, _ = expected(p[:, 0], p[:, 1], np.ones(n, bool), nx, ny, sd, 0.0)
        assert np.array_equal(final.cpu().numpy(), want)
