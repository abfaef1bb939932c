"""Whole steps and the calls that a step is made of, on one simulation."""
import numpy as np
import pytest

from zpic_gb300._zc import PART_DTYPE, CudaSim

pytestmark = pytest.mark.gpu


def _sim(filt, deterministic):
    nx, ny = 40, 24
    rng = np.random.default_rng(7)
    p = np.zeros(4 * nx * ny, dtype=PART_DTYPE)
    p["ix"], p["iy"] = rng.integers(0, nx, p.size), rng.integers(0, ny, p.size)
    p["x"], p["y"] = rng.random((2, p.size), dtype=np.float32)
    for u in ("ux", "uy", "uz"):
        p[u] = (0.4 * rng.standard_normal(p.size)).astype(np.float32)
    s = CudaSim((nx, ny), (0.1 * nx, 0.1 * ny), 0.06, deterministic=deterministic)
    s.add_species(-1.0, -0.25, (4, 1), p)
    if filt:
        s.set_smooth(*filt)
    return s


# no filter, one that the fused field phase takes, one that it leaves to the
# separate kernels
@pytest.mark.parametrize("filt", [None, ("compensated", 2, "binomial", 1), ("compensated", 5, "compensated", 5)])
@pytest.mark.parametrize("deterministic", [False, True])
def test_step_after_a_push_by_itself(filt, deterministic):
    """A push by itself leaves its deposits in the current that the next step
    starts from: that step has to clear them.  (Float sums in another order:
    1e-5, as against the oracle.)"""
    a, b = _sim(filt, deterministic), _sim(filt, deterministic)
    for s in (a, b):
        s.step(2)
        s.spec_advance(0)
    b.current_zero()
    for s in (a, b):
        s.step(1)
    for f in ("J", "E", "B"):
        x, y = getattr(a, f)(), getattr(b, f)()
        if deterministic:
            assert np.array_equal(x, y), f
        else:
            assert np.abs(x - y).max() <= 1e-5 * np.abs(y).max(), f
    a.close()
    b.close()
