"""A gradient on a GPU with little memory free: the states that a run may keep
to save recomputation leave room for what it cannot do without."""
import numpy as np
import pytest
import torch

from zpic_gb300.adjoint import AdjointSim

pytestmark = pytest.mark.gpu


def test_kept_states_leave_room_for_checkpoints():
    """4 million particles, segments of 16 steps (2.05 GB of states): four
    segments' states are within the 8 GiB that a run keeps, the engine starts
    with two, and 4.3 GB are free: the other two would fit, but then not all of
    the four checkpoints of 128 MB."""
    n, K, steps = 4_000_000, 16, 64
    rng = np.random.default_rng(2)
    st = [rng.integers(0, 64, n), rng.integers(0, 64, n), rng.random(n), rng.random(n)]
    st += [0.05 * rng.standard_normal(n) for _ in range(3)] + [np.ones(n)]
    sim = AdjointSim((64, 64), (6.4, 6.4), 0.05, n, -1e-3, checkpoint_every=K)
    sim.set_state(*st)
    free, _ = torch.cuda.mem_get_info()
    rest = torch.empty(free - 4_300_000_000, dtype=torch.uint8, device="cuda")
    assert 4.2e9 < torch.cuda.mem_get_info()[0] < 4.4e9
    L, _ = sim.forward(steps)
    g = sim.backward()
    del rest
    torch.cuda.empty_cache()
    # the same run with all the memory (float sums in another order)
    sim.set_state(*st)
    assert abs(sim.forward(steps)[0] - L) <= 1e-3 * L
    h = sim.backward()
    for k in g:
        assert np.linalg.norm(g[k] - h[k]) <= 1e-2 * np.linalg.norm(h[k]), k
    sim.close()
