"""Deterministic deposits: the lanes' running integer sums give the same bits
whatever tiles (and so runs and lanes) hold the particles, over the charges
that the sums of two parts take and those that go particle by particle."""
import numpy as np
import pytest

from test_gpu_push_paths import _parts
from zpic_gb300._zc import CudaSim

pytestmark = pytest.mark.gpu


def _sim(nx, ny, ppc, q, tile, fast):
    s = CudaSim((nx, ny), (0.1 * nx, 0.1 * ny), 0.06, tile=tile, deterministic=True, fast_math=fast, sort_every=2)
    s.add_species(-1.0, q, (max(ppc, 1), 1), _parts(nx, ny, ppc, 0.3, 4))
    return s


# a lane's sums cut after 512 particles (4700 a cell), by every cell change,
# by holes; the largest charge of two parts (5.33), the first beyond (a charge
# is refused where so many particles a tile could overflow the tile's sums)
@pytest.mark.parametrize("nx,ny,ppc,q", [
    (8, 8, 4700, -2.0**-32), (24, 40, 5, -0.2), (35, 17, 1, 0.5), (16, 16, 4, -5.3), (16, 16, 4, -5.4),
    (24, 24, 4, 8.0)])
@pytest.mark.parametrize("fast", [False, True])
def test_tiles_give_the_same_bits(nx, ny, ppc, q, fast):
    out = []
    for tile in ((8, 8), (16, 16), (32, 32)):
        s = _sim(nx, ny, ppc, q, tile, fast)
        for _ in range(3):  # (not split over a cluster, as a step of so few tiles would be)
            s.current_zero()
            s.spec_advance(0)
            s.current_update()
            s.emf_advance()
        out.append([getattr(s, f)() for f in ("E", "B", "J")])
        s.close()
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert np.array_equal(a, b)


def test_large_charge_scales():
    # contributions in proportion to the charge (a power of two), rounded to 2^-40
    J = []
    for q in (1.0, 16.0):
        s = _sim(24, 24, 6, q, (16, 16), False)
        s.current_zero()
        s.spec_advance(0)
        s.current_update()
        J.append(s.J() / q)
        s.close()
    assert np.abs(J[1] - J[0]).max() <= 1e-6 * np.abs(J[0]).max()
