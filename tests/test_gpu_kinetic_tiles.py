"""Deterministic kinetic energies are the exact sum of their terms, rounded once:
the same bits whatever tiles, runs and spill lists hold the particles, with
terms of many binades (see test_gpu_kinetic_bits)."""
import numpy as np
import pytest

from zpic_gb300._zc import PART_DTYPE, CudaSim

pytestmark = pytest.mark.gpu


def _run(tile, slack, seed, hot, steps=5):
    nx, ny, n = 64, 48, 30000
    rng = np.random.default_rng(1)
    p = np.zeros(n, dtype=PART_DTYPE)
    # most of them in a few cells, from where they spread over tiles with little room
    p["ix"], p["iy"] = rng.integers(20, 28, n), rng.integers(12, 20, n)
    p["ix"][:3000], p["iy"][:3000] = rng.integers(0, nx, 3000), rng.integers(0, ny, 3000)
    p["x"], p["y"] = rng.random((2, n), dtype=np.float32)
    for u in ("ux", "uy", "uz"):
        p[u] = rng.choice([-1, 1], n) * 10.0 ** rng.uniform(-6, hot, n)
    s = CudaSim((nx, ny), (0.1 * nx, 0.1 * ny), 0.06, tile=tile, deterministic=True, tile_slack=slack, sort_every=2)
    s.add_species(-1.0, -1e-5, (10, 1), p[np.random.default_rng(seed).permutation(n)])
    rows = []
    for _ in range(steps):
        s.step(1)
        rows.append(s.energy()[1][0])
    parts = np.sort(s.particles(0), order=["ix", "iy", "x", "y", "ux", "uy", "uz"])
    s.close()
    return rows, parts


@pytest.mark.parametrize("hot", [0.0, 1.5])
def test_bits_do_not_depend_on_tiles_or_spills(hot):
    ref, parts = _run((16, 16), 0.5, 0, hot)
    for tile, slack, seed in (((16, 16), 0.0, 1), ((8, 8), 0.0, 2), ((8, 8), 0.0, 3), ((32, 16), 0.1, 4),
                              ((32, 32), 0.5, 5)):
        rows, p = _run(tile, slack, seed, hot)
        assert p.tobytes() == parts.tobytes()
        assert rows == ref, (tile, slack)
