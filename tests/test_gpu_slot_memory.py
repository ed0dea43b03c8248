"""Device memory of sparse species: a cell of n particles owns at most n + n/2 + 16
slots of two buffers of 20 bytes (and the side lists 1/16 of the slots, three
lists of 24 bytes).  An empty species owns 16 a cell, so loading may add the
difference; 64 MiB are allowed for the allocator's granules.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ppc", [1, 3, 7, 16, 100])
def test_slots_of_sparse_species(ppc):
    import torch
    from test_gpu_particles import make_pic, small_workload
    n = 1500 if ppc < 16 else 600
    w = small_workload(n, n, ppc)
    with make_pic(w) as pic:
        pic.synchronize()
        free0, _ = torch.cuda.mem_get_info()
        for s in range(2):
            pic.load_plasma(s, ppc, 2.0, 3 + s)
        pic.synchronize()
        free1, _ = torch.cuda.mem_get_info()
    per_slot = 2 * 20 + 3 * 24 / 16
    slots = 2 * n * n * (ppc + ppc // 2 + 16 - 16)
    assert free0 - free1 <= slots * per_slot + 2 ** 26, (free0 - free1) / (2 * n * n)
