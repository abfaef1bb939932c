"""Charge and phase-space densities against numpy sums of the same float32
contributions (em2d/particles.c:1289-1321, 1510-1632): what remains is the
order of the float32 sums, bounded by (terms of the value) x 2^-23 x (sum of
their magnitudes)."""
import numpy as np
import pytest

from zpic_gb300._zc import PART_DTYPE, CudaSim

pytestmark = pytest.mark.gpu
F = np.float32


def _sim(nx, ny, ppc, tile, seed=4):
    rng = np.random.default_rng(seed)
    p = np.zeros(nx * ny * ppc, dtype=PART_DTYPE)
    p["ix"], p["iy"] = rng.integers(0, nx, p.size), rng.integers(0, ny, p.size)
    p["x"], p["y"] = rng.random((2, p.size), dtype=F)
    for u in ("ux", "uy", "uz"):
        p[u] = (0.3 * rng.standard_normal(p.size)).astype(F)
    s = CudaSim((nx, ny), (0.1 * nx, 0.2 * ny), 0.05, tile=tile)
    s.add_species(-1.0, -0.25, (ppc, 1), p)
    return s, p


def _check(got, terms, shape):
    """terms: [(flat index, float32 values, mask)]"""
    n = int(np.prod(shape))
    total, mag, cnt = np.zeros(n), np.zeros(n), np.zeros(n)
    for k, v, m in terms:
        np.add.at(total, k[m], v[m].astype(np.float64))
        np.add.at(mag, k[m], np.abs(v[m].astype(np.float64)))
        np.add.at(cnt, k[m], 1)
    err = np.abs(got.astype(np.float64).ravel() - total)
    assert np.all(err <= (cnt + 1) * 2.0 ** -23 * mag), float((err - cnt * 2.0 ** -23 * mag).max())


# both windows and the plain path: positions (a window that follows the tile),
# momenta (the whole grid at once, and a grid too large for it), a range that
# leaves particles out, a reversed one, one column
@pytest.mark.parametrize("quants,n,rng", [
    (("x1", "u1"), (70, 33), ((0.0, 7.0), (-1.0, 1.0))), (("u2", "u3"), (128, 128), ((-1.0, 1.0), (-0.4, 0.9))),
    (("x1", "x2"), (200, 90), ((1.0, 5.5), (9.0, -1.0))), (("u1", "x2"), (40, 300), ((1.0, -1.0), (0.0, 7.0))),
    (("u1", "u2"), (300, 300), ((-1.0, 1.0), (-1.0, 1.0))), (("u3", "u1"), (1, 2), ((-1.0, 1.0), (-1.0, 1.0)))])
@pytest.mark.parametrize("nx,ny,ppc,tile", [(70, 35, 5, (16, 16)), (33, 8, 40, (32, 16))])
def test_phasespace(quants, n, rng, nx, ny, ppc, tile):
    s, p = _sim(nx, ny, ppc, tile)
    got = s.phasespace(0, quants, n, rng)
    dx, dy = F(F(0.1 * nx) / F(nx)), F(F(0.2 * ny) / F(ny))
    val = {"x1": (p["x"] + p["ix"].astype(F)) * dx, "x2": (p["y"] + p["iy"].astype(F)) * dy, "u1": p["ux"],
           "u2": p["uy"], "u3": p["uz"]}
    at, w = [], []
    for a in range(2):
        lo, hi = F(rng[a][0]), F(rng[a][1])
        f = (val[quants[a]] - lo) * (F(n[a]) / (hi - lo))
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


@pytest.mark.parametrize("nx,ny,ppc,tile", [(70, 35, 5, (16, 16)), (33, 8, 40, (32, 16)), (9, 9, 1, (8, 8))])
def test_charge(nx, ny, ppc, tile):
    s, p = _sim(nx, ny, ppc, tile)
    got = s.charge(0)
    terms, row = [], nx + 1
    for c2 in (0, 1):
        for c1 in (0, 1):
            v = (p["x"] if c1 else F(1) - p["x"]) * (p["y"] if c2 else F(1) - p["y"]) * F(-0.25)
            i, j = (p["ix"] + c1).astype(np.int64), (p["iy"] + c2).astype(np.int64)
            every = np.ones(p.size, dtype=bool)
            terms.append((i + row * j, v, every))
            # the grid's first column and row also hold the last one's (periodic)
            terms.append((row * j, v, i == nx))
            terms.append((i, v, j == ny))
            terms.append((0 * i, v, (i == nx) & (j == ny)))
    _check(got, terms, (ny + 1, nx + 1))
    s.close()
