"""A window injection provider that fails (made on the host: it raises) leaves
every species as the step's push left it: what is read afterwards is what a run
whose provider had no particles for that species holds."""
import numpy as np
import pytest

from gpu_util import canon
from zpic_gb300._zc import PART_DTYPE, CudaSim, ZcError

pytestmark = pytest.mark.gpu

NX, NY, DX, DT = 40, 24, 0.1, 0.06


def _sim(nsp, provider):
    s = CudaSim((NX, NY), (NX * DX, NY * DX), DT, deterministic=True)  # (two runs are compared bit by bit)
    for k in range(nsp):
        rng = np.random.default_rng(k)
        p = np.zeros(3 * NX * NY, dtype=PART_DTYPE)
        p["ix"], p["iy"] = rng.integers(0, NX, p.size), rng.integers(0, NY, p.size)
        p["x"], p["y"] = rng.random((2, p.size), dtype=np.float32)
        for u in ("ux", "uy", "uz"):
            p[u] = (0.3 * rng.standard_normal(p.size)).astype(np.float32)
        s.add_species(-1.0 if k % 2 else 1.0, 1e-3, (3, 1), p)
    s.set_moving_window()
    if provider:
        s.set_injector(provider)
    return s


def _column(n_move):
    p = np.zeros(NY, dtype=PART_DTYPE)
    p["ix"], p["iy"] = NX - 1, np.arange(NY)
    p["x"] = p["y"] = 0.25
    return p


# all species in one launch (2 species), one launch each (9); the first or
# another species fails, or there is no provider at all
@pytest.mark.parametrize("nsp,bad", [(2, 0), (2, 1), (9, 0), (2, None)])
def test_species_after_a_failed_injection(nsp, bad):
    broken = [True]

    def failing(k, n_move):
        if broken[0] and k == bad:
            raise RuntimeError("no particles")
        return _column(n_move)

    def empty(k, n_move):
        if broken[0] and (bad is None or k == bad):
            return np.zeros(0, dtype=PART_DTYPE)
        return _column(n_move)

    a, b = _sim(nsp, None if bad is None else failing), _sim(nsp, empty)
    for s in (a, b):
        s.step(1)  # 0.06 of a cell of 0.1: the window has not moved
        assert s.info()["n_move"] == 0
    before = [a.count(k) for k in range(nsp)]
    with pytest.raises(ZcError) as exc:
        a.step(1)
    assert exc.value.status == (7 if bad is None else 1)
    b.step(1)
    # species behind the failing one: pushed with it, or (a launch each) not yet
    together = nsp <= 8
    for k in range(nsp if together else bad + 1):
        assert a.count(k) == b.count(k), k
        assert np.array_equal(canon(a.particles(k)), canon(b.particles(k))), k
    if not together:
        assert [a.count(k) for k in range(bad + 1, nsp)] == before[bad + 1:]
    # and the run goes on
    broken[0] = False
    if bad is None:
        a.set_injector(empty)
    a.step(4)
    for k in range(nsp):
        p = a.particles(k)
        assert p.size == a.count(k) and np.all((p["ix"] >= 0) & (p["ix"] < NX) & (p["iy"] >= 0) & (p["iy"] < NY))
    a.close()
    b.close()
