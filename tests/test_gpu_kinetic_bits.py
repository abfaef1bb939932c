"""Deterministic kinetic energies with terms of many binades (a cold plasma with
a few fast particles): a tile's sum needs more bits than a double has, so it is
rounded once, from its exact integers, whatever parts of the tile, and so slots
and runs, held which particle."""
import numpy as np
import pytest

from zpic_gb300._zc import PART_DTYPE, CudaSim

pytestmark = pytest.mark.gpu


def _sim(nx, ny, ppc, nsp, seed):
    s = CudaSim((nx, ny), (0.1 * nx, 0.1 * ny), 0.06, tile=(16, 16), deterministic=True, sort_every=3)
    for k in range(nsp):
        rng = np.random.default_rng(k)
        p = np.zeros(nx * ny * ppc, dtype=PART_DTYPE)
        cell = np.arange(p.size) // ppc
        p["ix"], p["iy"] = cell % nx, cell // nx
        p["x"], p["y"] = rng.random((2, p.size), dtype=np.float32)
        for u in ("ux", "uy", "uz"):
            p[u] = rng.choice([-1, 1], p.size) * 10.0 ** rng.uniform(-6, 0.5, p.size)
        # the same particles, in an order of this run's own
        s.add_species(-1.0, -1e-4, (ppc, 1), p[np.random.default_rng(seed).permutation(p.size)])
    return s


# tiles in 8 parts, in 4, and ragged ones in 8
@pytest.mark.parametrize("nx,ny,ppc,nsp", [(64, 48, 64, 1), (128, 128, 16, 2), (40, 24, 9, 3)])
def test_split_tiles_give_the_bits_of_whole_ones(nx, ny, ppc, nsp):
    kin = []
    for seed in (1, 2, 3):
        s = _sim(nx, ny, ppc, nsp, seed)
        s.history_enable(8)
        rows = []
        for _ in range(6):
            s.step(1)
            rows.append(s.energy()[1])
        assert np.array_equal(s.history()[:6, 6:], np.array(rows))
        kin.append(rows)
        s.close()
    whole = _sim(nx, ny, ppc, nsp, 4)
    for n in range(6):
        whole.current_zero()
        for k in range(nsp):
            whole.spec_advance(k)
        whole.current_update()
        whole.emf_advance()
        for rows in kin:
            assert np.array_equal(rows[n], whole.energy()[1]), n
    whole.close()
