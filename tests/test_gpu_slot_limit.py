"""Loads that a species cannot hold are refused with the state as it was: more
slots than 32-bit indices reach (72,900 cells of 40,000 particles want 4.4e9, whose
32-bit sum is 8e7), and a cell beyond the per-cell limit.  Where the device's
memory does not hold the larger buffers the species is left empty, and the
context usable.
"""
import numpy as np
import pytest

from test_gpu_particles import export_state, make_pic, multiset, small_workload

pytestmark = pytest.mark.gpu


def test_refused_loads_keep_the_particles():
    import pic_b200 as P
    w = small_workload(270, 270, 4)
    with make_pic(w) as pic:
        for s in range(2):
            pic.load_plasma(s, 4, 2.0, 7 + s)
        pic.step(0)
        before = [multiset(export_state(pic, s)) for s in range(2)]
        with pytest.raises(P.PicError) as e:
            pic.load_plasma(0, 40000, 2.0, 1)
        assert e.value.status == -3 and "slots" in str(e.value)
        with pytest.raises(P.PicError) as e:
            pic.load_plasma(1, 50000, 2.0, 1)
        assert e.value.status == -3
        for s in range(2):
            assert np.array_equal(multiset(export_state(pic, s)), before[s])
        pic.step(1)
        assert 0 < pic.count(0) <= len(before[0])


def test_load_that_does_not_fit_the_memory():
    import torch
    import pic_b200 as P
    w = small_workload(600, 600, 4)
    with make_pic(w) as pic:
        pic.load_plasma(0, 4, 2.0, 7)
        pic.load_plasma(1, 4, 0.026, 8)
        pic.step(0)
        free, _ = torch.cuda.mem_get_info()
        hold = torch.empty(free - (1 << 30), dtype=torch.uint8, device="cuda")
        with pytest.raises(P.PicError):
            pic.load_plasma(0, 400, 2.0, 9)  # 360,000 cells x 616 slots x 40 bytes
        assert pic.count(0) == 0 and pic.count(1) > 0
        pic.step(1)
        del hold
        torch.cuda.empty_cache()
        pic.load_plasma(0, 20, 2.0, 9)
        pic.step(2)
        assert pic.count(0) > 19 * 600 * 600
