"""The float64 field advance of a large grid, a kernel each, against the one
kernel of a small one: a wave on a grid that repeats it in y advances in every
copy as on one copy, bit by bit."""
import numpy as np
import pytest

from zpic_gb300.adjoint import AdjointSim

pytestmark = pytest.mark.gpu


def _run(nx, ny, E, B, copies, particles):
    tile = lambda a, n: np.concatenate([a] * n)  # noqa: E731
    ix, iy, rest = particles
    iy = np.concatenate([iy + c * ny for c in range(copies)])
    s = AdjointSim((nx, ny * copies), (0.125 * nx, 0.125 * ny * copies), 0.05, iy.size, -0.1, checkpoint_every=3,
                   precision="float64")
    s.set_state(tile(ix, copies), iy, *[tile(v, copies) for v in rest], E=np.concatenate([E] * copies, axis=1),
                B=np.concatenate([B] * copies, axis=1))
    s.forward(7)
    out = s.state()
    s.close()
    return out


# 65536 cells or more are advanced by a kernel each: just that many, ragged ones
@pytest.mark.parametrize("nx,ny,copies", [(128, 64, 8), (257, 17, 16), (1024, 3, 22)])
@pytest.mark.parametrize("n", [0, 50])
def test_large_grid_repeats_small_one(nx, ny, copies, n):
    rng = np.random.default_rng(nx)
    E, B = rng.standard_normal((2, 3, ny, nx)) * 0.1
    # particles apart from each other, so that no node sums two of them
    cell = rng.choice(np.arange(0, nx * ny, 8), n, replace=False) if n else np.zeros(0, dtype=np.int64)
    cell = cell[(cell // nx) % 4 == 0] if ny > 4 else cell[cell // nx == 0]
    particles = (cell % nx, cell // nx, [rng.random(cell.size) * 0.2 + 0.2 for _ in range(2)]
                 + [0.01 * rng.standard_normal(cell.size) for _ in range(3)] + [np.ones(cell.size)])
    a, b = _run(nx, ny, E, B, 1, particles), _run(nx, ny, E, B, copies, particles)
    assert nx * ny < 65536 <= nx * ny * copies
    for f in ("E", "B"):
        for c in range(copies):
            assert np.array_equal(b[f][:, c * ny:(c + 1) * ny], a[f]), (f, c)
