"""A density's device memory: small buffers stay with the simulation, large ones
are given back when the call returns."""
import numpy as np
import pytest
import torch

from zpic_gb300._zc import PART_DTYPE, CudaSim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(64, 64), (4096, 4096), (4096, 4097), (16384, 8192)])
def test_memory_after_a_phasespace(n):
    p = np.zeros(64, dtype=PART_DTYPE)
    p["ix"], p["x"], p["y"], p["ux"] = np.arange(64) % 16, 0.25, 0.5, 0.125
    s = CudaSim((16, 16), (16.0, 16.0), 0.5)
    s.add_species(-1.0, -0.25, (1, 1), p)
    calls = [(("u1", "u2"), n, ((-1.0, 1.0), (-1.0, 1.0))), (("u1", "u2"), (8, 8), ((-1.0, 1.0), (-1.0, 1.0)))]
    small = s.phasespace(0, *calls[1])
    free, _ = torch.cuda.mem_get_info()
    big = s.phasespace(0, *calls[0])
    assert free - torch.cuda.mem_get_info()[0] <= (66 << 20)
    assert np.array_equal(s.phasespace(0, *calls[1]), small)  # after the buffer went, and came again
    assert np.array_equal(s.phasespace(0, *calls[0]), big) and big.sum() == -16.0
    s.close()
