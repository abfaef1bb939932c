"""The two ways a step pushes its species: all together with tiles split into
parts (small grids), or one launch a species.  zc_step takes the first where
its rule says so, zc_spec_advance always the second; in deterministic mode
both give the same bits whatever holds which particle."""
import numpy as np
import pytest

from gpu_util import canon
from zpic_gb300._zc import PART_DTYPE, CudaSim

pytestmark = pytest.mark.gpu


def _parts(nx, ny, ppc, uth, seed):
    rng = np.random.default_rng(seed)
    n = nx * ny * ppc
    p = np.zeros(n, dtype=PART_DTYPE)
    cell = np.arange(n) // max(ppc, 1)
    p["ix"], p["iy"] = cell % nx, cell // nx
    p["x"], p["y"] = rng.random((2, n), dtype=np.float32)
    for u in ("ux", "uy", "uz"):
        p[u] = uth * rng.standard_normal(n).astype(np.float32)
    return p


# few tiles and many particles (split 8 ways), ragged sizes, a tile of one
# column, no particles at all, one particle, more species than one launch
# takes, more tiles than the rule admits
@pytest.mark.parametrize("nx,ny,ppc,nsp,tile", [
    (16, 16, 64, 1, (16, 16)), (32, 24, 4, 2, (16, 16)), (33, 17, 9, 3, (16, 16)), (40, 40, 1, 2, (8, 8)),
    (70, 35, 7, 2, (32, 16)), (64, 64, 0, 2, (32, 32)), (50, 20, 3, 9, (16, 8)), (400, 420, 1, 1, (16, 16))])
@pytest.mark.parametrize("fast", [False, True])
def test_together_matches_one_by_one(nx, ny, ppc, nsp, tile, fast):
    sims = []
    for _ in range(2):
        s = CudaSim((nx, ny), (0.1 * nx, 0.1 * ny), 0.06, tile=tile, deterministic=True, fast_math=fast, sort_every=3)
        for k in range(nsp):
            p = _parts(nx, ny, ppc, 0.4, 10 + k)
            if k == 1 and nsp == 3:
                p = p[:1]
            s.add_species(-1.0 if k % 2 else 1.5, -0.05, (max(ppc, 1), 1), p)
        sims.append(s)
    a, b = sims
    for _ in range(7):
        a.step(1)
        b.current_zero()
        for k in range(nsp):
            b.spec_advance(k)
        b.current_update()
        b.emf_advance()
    for f in ("E", "B", "J"):
        assert np.array_equal(getattr(a, f)(), getattr(b, f)()), f
    ea, eb = a.energy(), b.energy()
    # the same terms, summed over other partials (double sums of exact parts)
    np.testing.assert_allclose(ea[1], eb[1], rtol=1e-13)
    for k in range(nsp):
        assert np.array_equal(canon(a.particles(k)), canon(b.particles(k))), k
    a.close()
    b.close()
