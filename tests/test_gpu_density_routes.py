"""Densities over two positions on both sides of every line of the rule that
takes them through shared-memory windows or straight to the grid, both ways
round, against numpy sums (as in test_gpu_densities)."""
import numpy as np
import pytest

from test_gpu_densities import F, _check, _sim

pytestmark = pytest.mark.gpu


# a tile of 16 x 16 cells spans sx x sy values: (1.5, 1.6) and (1.4, 4) window,
# (1.6, 4) grid, (1.4, 1.4) window; (2, 11) grid and (2, 13) window; 32 particles
# a cell always the window
@pytest.mark.parametrize("ppc,span", [(3, (1.5, 1.6)), (3, (1.4, 4.0)), (3, (1.6, 4.0)), (3, (1.4, 1.4)),
                                      (3, (2.0, 11.0)), (3, (2.0, 13.0)), (3, (5.0, 5.0)), (32, (5.0, 5.0))])
@pytest.mark.parametrize("swap", [False, True])
def test_two_positions(ppc, span, swap):
    nx, ny = 70, 35
    s, p = _sim(nx, ny, ppc, (16, 16))
    n = [int(round(span[0] * nx / 16)), int(round(span[1] * ny / 16))]
    rng = [(0.3, 0.1 * nx), (0.0, 0.2 * ny - 0.4)]  # (particles on both sides of the range)
    dx, dy = F(F(0.1 * nx) / F(nx)), F(F(0.2 * ny) / F(ny))
    val = [(p["x"] + p["ix"].astype(F)) * dx, (p["y"] + p["iy"].astype(F)) * dy]
    names = ["x1", "x2"]
    if swap:
        n, rng, val, names = n[::-1], rng[::-1], val[::-1], names[::-1]
    got = s.phasespace(0, names, n, rng)
    at, w = [], []
    for a in range(2):
        lo, hi = F(rng[a][0]), F(rng[a][1])
        f = (val[a] - lo) * (F(n[a]) / (hi - lo))
        i = np.trunc(f + F(0.5)).astype(np.int64)
        at.append(i)
        w.append(f - i.astype(F) + F(0.5))
    terms = []
    for c2 in (0, 1):
        for c1 in (0, 1):
            i1, i2 = at[0] + c1, at[1] + c2
            v = (w[0] if c1 else F(1) - w[0]) * (w[1] if c2 else F(1) - w[1]) * F(-0.25)
            ok = (i1 >= 0) & (i1 < n[0]) & (i2 >= 0) & (i2 < n[1])
            terms.append((np.where(ok, i1 + n[0] * i2, 0), v, ok))
    _check(got, terms, (n[1], n[0]))
    s.close()
