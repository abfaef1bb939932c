"""The 1-D step as one launch for several steps against the same step as two
kernels (what a profiled simulation runs): equal particle counts, counters and
pushed particles; fields, current and energies within the 1e-5 that separates
float32 deposits summed in another order (as against the oracle)."""
import numpy as np
import pytest

from zpic_gb300 import em1d_gpu

pytestmark = pytest.mark.gpu


def _sim(nx, species, mode, smooth, sort, ctas):
    kw = {"window": dict(moving_window=True), "open": dict(open_fields=True, open_particles=True),
          "periodic": {}}[mode]
    s = em1d_gpu.CudaSim1D(nx, nx * 0.02, 0.019, sort_every=sort, push_ctas=ctas, **kw)
    for k, (ppc, n, density) in enumerate(species):
        rng = np.random.default_rng(k)
        p = np.zeros(n, dtype=em1d_gpu.PART_DTYPE)
        p["ix"] = np.sort(rng.integers(0, nx, n))
        p["x"] = rng.random(n, dtype=np.float32)
        for u in ("ux", "uy", "uz"):
            p[u] = (0.3 * rng.standard_normal(n)).astype(np.float32)
        s.add_species(-1.0 if k == 0 else 1.0, (-1.0 if k == 0 else 1.0) / ppc, ppc, p, ufl=(0.0, 0.1, -0.1),
                      density=density)
    if smooth:
        s.set_smooth(*smooth)
    s.add_laser(0.8 * nx * 0.02, 1.0, 5.0, fwhm=0.2 * nx * 0.02, polarization=0.5)
    return s


# particles: none, one, less than a CTA each, several rounds of a CTA's slots,
# more than fit (the two kernels then); columns: larger than a CTA, cut by the
# profile; the fewest cells; passes: none, the most
@pytest.mark.parametrize("nx,species,mode,smooth,sort,ctas", [
    (4, [(1, 1, ("uniform", 0.0, 0.0))], "periodic", None, 0, 0),
    (50, [(8, 0, ("uniform", 0.0, 0.0))], "window", ("binomial", 1), 0, 0),
    (200, [(16, 3000, ("step", 3.3, 0.0)), (4, 777, ("slab", 1.0, 4.25))], "window", ("compensated", 4), 5, 0),
    (200, [(16, 3000, ("uniform", 0.0, 0.0)), (4, 777, ("empty", 0.0, 0.0))], "open", ("compensated", 15), 0, 4),
    (1000, [(128, 90000, ("step", 20.007, 0.0))], "window", ("compensated", 4), 0, 0),
    (1000, [(2500, 4000, ("slab", 19.9, 20.2))], "window", None, 3, 16),
    (333, [(64, 40000, ("uniform", 0.0, 0.0)), (64, 40000, ("uniform", 0.0, 0.0))], "periodic", ("binomial", 2), 7, 4),
    (64, [(2, 200000, ("uniform", 0.0, 0.0))], "periodic", ("binomial", 1), 0, 16)])
def test_run_matches_two_kernels(nx, species, mode, smooth, sort, ctas):
    a, b = (_sim(nx, species, mode, smooth, sort, ctas) for _ in range(2))
    b.set_profile(True)
    for n, wait in ((1, True), (2, False), (16, False), (21, True), (1, False), (3, True)):
        a.step(n, wait=wait)
        b.step(n)
    assert a.info() == b.info()
    for k in range(len(species)):
        assert a.count(k) == b.count(k) and a.pushed(k) == b.pushed(k)
    for f in ("E", "B", "J"):
        x, y = getattr(a, f)(), getattr(b, f)()
        assert np.abs(x - y).max() <= 1e-5 * max(np.abs(y).max(), 1e-30), f
    ea, eb = a.energy(), b.energy()
    np.testing.assert_allclose(ea[0], eb[0], rtol=1e-5, atol=1e-5 * max(ea[0].max(), 1e-30))
    np.testing.assert_allclose(ea[1], eb[1], rtol=1e-5)
    a.close()
    b.close()
