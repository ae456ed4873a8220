"""One environment: the walk that keeps its row and makes its draws 128 steps ahead, against the oracle -- around those 128 steps, with every option, on worlds in
shared and in global memory, and on tables with ties, infinities and entries that are no numbers."""
import numpy as np
import pytest

from test_gpu_engines import world
from test_gpu_parity import pair

pytestmark = pytest.mark.gpu


def assert_same(gpu, cpu, what):
    assert [int(v[0]) for v in gpu.get_state()] == [int(v[0]) for v in cpu.get_state()], what
    assert np.array_equal(gpu.get_q(), cpu.get_q(), equal_nan=True), what
    a, b = gpu.get_stats(), cpu.get_stats()
    assert (a.goals, a.timeouts, a.conflicts, a.epsilon, a.device_error) == (b.goals, b.timeouts, b.conflicts, b.epsilon, 0), what


@pytest.mark.parametrize("w,h", [(10, 10), (3, 2), (1, 13011), (170, 160)])
@pytest.mark.parametrize("kw", [{}, {"eps_kind": 1, "eps0": 1.0, "eps_decay": 0.99}, {"eps_kind": 2, "eps0": 1.0, "eps_decay": 0.9, "legacy_clamp": 1}, {"start_mode": 0, "max_steps": 0}])
def test_around_the_draws_made_ahead(pkg, orc, w, h, kw):
    cfg = world(pkg, w, h, 1, num_goals=1, env_offset=7, **kw)
    gpu, cpu = pair(pkg, orc, cfg)
    for k in np.flatnonzero(gpu.get_cells() == 1)[:9]:
        gpu.add_trap(int(k % w), int(k // w), -0.4); cpu.add_trap(int(k % w), int(k // w), -0.4)
    gpu.set_trace(True)
    for k in (1, 127, 128, 129, 400):
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "+%d" % k)
        assert [v[0] for v in gpu.get_trace()] == [v[0] for v in cpu.get_trace()]


@pytest.mark.parametrize("seed", range(6))
def test_rows_with_ties_infinities_and_no_numbers(pkg, orc, seed):
    rng = np.random.RandomState(seed)
    gpu, cpu = pair(pkg, orc, world(pkg, 9, 8, 1, num_goals=1, obstacle_p=0.1, max_steps=13, eps0=0.2, lr=0.5))
    q = rng.choice(np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, np.nan, -3.4e38, 1e-42], np.float32), (8, 9, 4))
    gpu.set_q(q); cpu.set_q(q)
    for k in (1, 1, 1, 20, 60):
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "+%d" % k)
