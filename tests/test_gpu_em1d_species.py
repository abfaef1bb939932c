"""A 1-D species takes memory for what its run can use."""
import numpy as np
import pytest
import torch

from zpic_gb300 import em1d_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,density", [({}, ("uniform", 0.0, 0.0)),
                                        ({"moving_window": True}, ("empty", 0.0, 0.0))])
def test_no_lattice_without_injection(kw, density):
    """The particles a cell only count where a window injects: a large number is
    as good as any elsewhere."""
    sims = []
    for ppc in (1, 400_000_000):
        p = np.zeros(100, dtype=em1d_gpu.PART_DTYPE)
        p["ix"], p["x"], p["ux"] = np.arange(100), 0.3, 0.1
        s = em1d_gpu.CudaSim1D(100, 10.0, 0.09, **kw)
        free, _ = torch.cuda.mem_get_info()
        s.add_species(-1.0, -1e-3, ppc, p, density=density)
        assert free - torch.cuda.mem_get_info()[0] < 64 << 20
        s.step(4)
        sims.append(s)
    assert sims[0].count(0) == sims[1].count(0)
    assert np.allclose(sims[0].E(), sims[1].E(), rtol=0, atol=1e-5 * np.abs(sims[0].E()).max())
    for s in sims:
        s.close()
