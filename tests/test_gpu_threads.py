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
