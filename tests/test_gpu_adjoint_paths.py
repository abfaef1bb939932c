"""The float32 adjoint step (vector reductions on the periodic grid, plain ones
under a window) against the float64 engine, and a reverse sweep that walks kept
states against one that recomputes them."""
import numpy as np
import pytest

from zpic_gb300.adjoint import AdjointSim

pytestmark = pytest.mark.gpu

KEYS = ("w", "x", "y", "ux", "uy", "uz", "E", "B")


def _inputs(nx, ny, n, cols, u, seed=5):
    rng = np.random.default_rng(seed)
    f32 = lambda a: a.astype(np.float32).astype(np.float64)  # noqa: E731
    # in-cell positions away from the edges and the half cell, where a gradient's pieces meet
    pos = lambda: f32(rng.choice([0.05, 0.55], n) + 0.4 * rng.random(n))  # noqa: E731
    st = [rng.integers(0, nx, n), rng.integers(0, ny, n), pos(), pos()]
    st += [f32(u * rng.standard_normal(n)) for _ in range(3)] + [f32(1 + 0.3 * rng.random(n))]
    return st, [f32(0.05 * rng.standard_normal((3, ny, cols))) for _ in range(2)]


def _gradient(nx, ny, inputs, steps, K, precision, window=False, passes=()):
    st, fields = inputs
    sim = AdjointSim((nx, ny), (nx * 0.1, ny * 0.1), 0.05, st[0].size, -0.1, checkpoint_every=K, precision=precision,
                     moving_window=window)
    sim.set_smooth(passes)
    for _ in range(2):  # the second run starts from used buffers
        sim.set_state(*st, E=fields[0], B=fields[1])
        L, kin = sim.forward(steps)
        g = sim.backward()
    sim.close()
    return g | {"L": np.array([L]), "kin": np.array([kin])}


# rounding (6e-8) of some 100 operations a step, in 3 steps: 1e-4 is ten times that
@pytest.mark.parametrize("nx,ny,n,window,passes", [
    (2, 2, 1, False, ()), (3, 2, 31, False, ()), (2, 5, 33, False, [(0.25, 0.5)]), (33, 7, 5000, False, ()),
    (16, 16, 0, False, ()), (40, 24, 4097, False, [(0.25, 0.5), (-0.1, 1.2)]), (40, 24, 4097, True, ()),
    (9, 6, 200, True, [(0.25, 0.5)])])
def test_float32_matches_float64(nx, ny, n, window, passes):
    inputs = _inputs(nx, ny, n, nx + 3 if window else nx, 0.4)
    a, b = (_gradient(nx, ny, inputs, 3, 2, p, window, passes) for p in ("float32", "float64"))
    for k in KEYS + ("L", "kin"):
        assert np.linalg.norm(a[k] - b[k]) <= 1e-4 * np.linalg.norm(b[k]) + 1e-12, k


def test_recomputed_segments_match_kept_ones():
    """2 million particles: two segments of 70 steps' states are more than the 8 GiB
    that a run keeps, so the first is recomputed; of 10 steps, all are kept in 64
    bits.  Float64: rounding (1e-16) of 75 steps of a sensitive system (float32
    differs by 2e-3 from run to run); float32: the 1e-2 of the full-size gradient."""
    inputs = _inputs(64, 64, 2_000_000, 64, 0.05)
    kept = _gradient(64, 64, inputs, 75, 10, "float64")
    for precision, tol in (("float64", 1e-9), ("float32", 1e-2)):
        a = _gradient(64, 64, inputs, 75, 70, precision)
        for k in KEYS + ("L", "kin"):
            assert np.linalg.norm(a[k] - kept[k]) <= tol * np.linalg.norm(kept[k]), (precision, k)
