"""Solve times of ensembles of few small instances, whose many blocks have little
to sum.  The bounds are what the batched solve took on a B200 when an instance's
first block alone summed (1 instance of 16^2 cells 247 us, 3 of them 237, 2 of
32^2 246), with a sixth more for the clock; every block reading every
partial sum in turn took 461, 295 and 348.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,limit_us", [(16, 1, 288.0), (16, 3, 277.0), (32, 2, 287.0)])
def test_solve_time_of_few_small_instances(n, count, limit_us):
    import pic_b200 as P
    import pic_configs as C
    cfgs = [P.make_config(n, n, n * 2.5e-4, n * 2.5e-4, 5e-11, C._species(n, n, 8, 1e15),
                          C.wall_rects(n, n, left=50.0 + k), b0=0.01) for k in range(count)]
    with P.Ensemble(cfgs) as E:
        for k in range(count):
            for s in range(2):
                E[k].load_plasma(s, 8, (2.0, 0.026)[s], 2 * k + s)
        us = []
        for it in range(12):
            E.step(it)
            us.append(E.timing()[1] * 1e3)
        assert all(E[k].poisson_stats()[1] <= 1e-8 for k in range(count))
    assert np.median(us[3:]) <= limit_us, us
