"""The field phase of a step in one launch (fold, filter, Yee advance, external
fields) against the separate launches behind zc_current_update and
zc_emf_advance: the same bits in every cell, guard cells included.  The
current comes from deterministic deposits, so both start from one."""
import numpy as np
import pytest

from zpic_gb300._zc import PART_DTYPE, CudaSim

pytestmark = pytest.mark.gpu

# smallest grid it takes, its output tile (32 x 16) met exactly, passed by one,
# several wraps of the halo, tiles clear of the edges
SIZES = [(6, 6), (7, 31), (29, 13), (32, 16), (33, 17), (61, 45), (130, 70)]
FILTERS = [None, ("binomial", 1, "binomial", 1), ("compensated", 1, "none", 0), ("none", 2, "compensated", 2),
           ("compensated", 3, "binomial", 1), ("binomial", 4, "compensated", 3), ("compensated", 4, "none", 0)]


def _sim(nx, ny, filt, window, ext):
    s = CudaSim((nx, ny), (0.1 * nx, 0.1 * ny), 0.06, deterministic=True)
    rng = np.random.default_rng(nx + 100 * ny)
    p = np.zeros(3 * nx * ny, dtype=PART_DTYPE)
    p["ix"], p["iy"] = rng.integers(0, nx, p.size), rng.integers(0, ny, p.size)
    p["x"], p["y"] = rng.random((2, p.size), dtype=np.float32)
    for u in ("ux", "uy", "uz"):
        p[u] = rng.standard_normal(p.size).astype(np.float32)
    s.add_species(-1.0, -0.3, (3, 1), p)
    shape = (ny + 3, nx + 3, 3)
    if ext == "custom":
        s.set_ext_fld(E_type="custom", E_grid=rng.standard_normal(shape) * 0.1, B_type="uniform", B_0=(0.1, 0.2, 0.3))
    elif ext == "uniform":
        s.set_ext_fld(B_type="uniform", B_0=(0.0, -0.4, 0.3))
    if filt:
        s.set_smooth(*filt)
    if window:
        s.set_moving_window()
        s.set_device_injector(0, "uniform")
    return s


@pytest.mark.parametrize("window,ext", [(False, None), (False, "custom"), (True, None), (True, "uniform")])
@pytest.mark.parametrize("filt", FILTERS)
@pytest.mark.parametrize("nx,ny", SIZES)
def test_one_launch_matches_separate_ones(nx, ny, filt, window, ext):
    a, b = _sim(nx, ny, filt, window, ext), _sim(nx, ny, filt, window, ext)
    for step in range(4):
        a.step(1)
        b.current_zero()
        b.spec_advance(0)
        b.current_update()
        b.emf_advance()
        for f in ("J", "E", "B", "E_part", "B_part"):
            x, y = getattr(a, f)(), getattr(b, f)()
            assert np.array_equal(x, y), (f, step, np.argwhere(x != y)[:5])
    # a call on the current by itself continues from the step's current
    a.current_update()
    b.current_update()
    if not filt:
        assert np.array_equal(a.J(), b.J())
    assert a.info()["n_move"] == b.info()["n_move"]
    a.close()
    b.close()
