"""Simulations are independent of each other: host threads that drive one each
get what a thread by itself gets."""
import threading

import numpy as np
import pytest

from zpic_gb300._zc import PART_DTYPE, CudaSim

pytestmark = pytest.mark.gpu


def _sim():
    # cells of size 1, positions and momenta in few binary digits: every
    # contribution to a density and every sum of them is exact
    nx, ny = 16, 16
    rng = np.random.default_rng(3)
    p = np.zeros(nx * ny, dtype=PART_DTYPE)
    p["ix"], p["iy"] = rng.integers(0, nx, p.size), rng.integers(0, ny, p.size)
    for x in ("x", "y"):
        p[x] = rng.integers(0, 8, p.size) / 8
    for u in ("ux", "uy", "uz"):
        p[u] = rng.integers(-32, 32, p.size) / 64
    s = CudaSim((nx, ny), (nx, ny), 0.5)
    s.add_species(-1.0, -0.25, (1, 1), p)
    return s


def test_phasespaces_of_different_sizes():
    """The windows of the two densities take 56 KB and 1 KB of shared memory."""
    calls = [(("u2", "u3"), (128, 112), ((-1.0, 1.0), (-1.0, 0.75))),
             (("x1", "u1"), (16, 16), ((0.0, 16.0), (-1.0, 1.0)))] * 4
    sims = [_sim() for _ in calls]
    alone = [s.phasespace(0, *c) for s, c in zip(sims, calls)]
    assert all(a.any() for a in alone)
    wrong = []

    def work(s, c, a):
        try:
            for _ in range(8000):
                if wrong:
                    return
                if not np.array_equal(s.phasespace(0, *c), a):
                    wrong.append(c[0])
        except Exception as e:
            wrong.append(e)

    threads = [threading.Thread(target=work, args=z) for z in zip(sims, calls, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s in sims:
        s.close()
    assert not wrong, wrong


def test_waiting_1d_steps_share_the_gpu():
    """Eight runs of a 1-D deck, stepped by a thread each that waits: after 32
    steps each has the particles and, within float sums in another order (1e-5,
    as against the oracle), the fields of a run by itself; and their steps take
    0.3 of the time of one run after another.  (Launches that fill the GPU, one
    a thread, queue: 0.77.  The bar lies between.)"""
    import time

    from zpic_gb300 import em1d_gpu

    def run():
        nx = 1000
        rng = np.random.default_rng(1)
        p = np.zeros(64 * nx, dtype=em1d_gpu.PART_DTYPE)
        p["ix"] = np.sort(rng.integers(0, nx, p.size))
        p["x"] = rng.random(p.size, dtype=np.float32)
        s = em1d_gpu.CudaSim1D(nx, 0.02 * nx, 0.019, moving_window=True)
        s.add_species(-1.0, -1.0 / 128, 128, p)
        s.set_smooth("compensated", 4)
        s.add_laser(16.0, 1.0, 5.0, fwhm=2.0)
        return s

    def threads(sims, calls):
        ts = [threading.Thread(target=lambda s: [s.step(16) for _ in range(calls)], args=(s,)) for s in sims]
        t0 = time.perf_counter()
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        return time.perf_counter() - t0

    alone, sims = run(), [run() for _ in range(8)]
    threads([alone], 2)
    threads(sims, 2)
    for s in sims:
        assert s.info() == alone.info() and s.count(0) == alone.count(0) and s.pushed(0) == alone.pushed(0)
        for f in ("E", "B", "J"):
            x, y = getattr(s, f)(), getattr(alone, f)()
            assert np.abs(x - y).max() <= 1e-5 * max(np.abs(y).max(), 1e-30), f
    one = min(threads([alone], 40) for _ in range(3))
    both = min(threads(sims, 40) for _ in range(3))
    for s in sims + [alone]:
        s.close()
    assert both <= 0.55 * 8 * one, (both, one)
