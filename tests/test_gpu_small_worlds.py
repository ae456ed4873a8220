"""Worlds of one block against the oracle: both sides of every number of threads, launches that end around the steps whose draws are made ahead, the largest grids, every
option."""
import numpy as np
import pytest

from test_gpu_engines import world
from test_gpu_parity import assert_same, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,n", [(9, 8, 2), (9, 8, 32), (20, 19, 33), (20, 19, 64), (20, 19, 65), (31, 33, 128), (31, 33, 129), (31, 33, 256), (31, 33, 257), (50, 62, 512), (50, 62, 513),
                                   (50, 62, 1024), (40, 20, 32), (60, 60, 32), (110, 110, 2), (4722, 1, 40), (1, 4723, 40), (83, 83, 1000), (80, 80, 500), (1, 6676, 32), (1, 6677, 32), (6429, 1, 500), (6430, 1, 500), (1, 6924, 1000), (1, 6925, 1000), (3, 2, 700)])
def test_worlds_of_one_block(pkg, orc, w, h, n):
    cfg = world(pkg, w, h, n, num_goals=1 if w * h < 100 else 3, obstacle_p=0.0 if w * h < 100 else 0.15, max_steps=29, env_offset=11)
    gpu, cpu = pair(pkg, orc, cfg)
    for k in (1, 3, 4, 5, 1, 1, 2, 31, 1, 32, 33, 130):
        gpu.set_trace(k in (5, 2, 33))                       # with and without the options
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "+%d" % k)
        assert k not in (5, 2, 33) or all(np.array_equal(a, b) for a, b in zip(gpu.get_trace(), cpu.get_trace()))
    a, b = gpu.get_stats(), cpu.get_stats()
    assert (a.conflicts, a.goals, a.timeouts, a.episodes, a.device_error) == (b.conflicts, b.goals, b.timeouts, b.episodes, 0)


@pytest.mark.parametrize("n", [20, 100, 500, 900])
@pytest.mark.parametrize("kw", [{"eps_kind": 2, "eps0": 1.0, "eps_decay": 0.9, "start_mode": 0}, {"eps_kind": 1, "eps0": 1.0, "eps_decay": 0.99},
                                {"eps_kind": 3, "eps0": 1.0, "eps_end": 0.1, "eps_steps": 60, "legacy_clamp": 1}])
def test_epsilons_traps_clamp_and_common_start(pkg, orc, n, kw):
    cfg = world(pkg, 41, 37, n, **kw)
    gpu, cpu = pair(pkg, orc, cfg)
    for k in np.flatnonzero(gpu.get_cells() == 1)[:40]:
        gpu.add_trap(int(k % 41), int(k // 41), -0.3); cpu.add_trap(int(k % 41), int(k // 41), -0.3)
    for k in (1, 33, 2, 64):
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "+%d" % k)
        a, b = gpu.get_stats(), cpu.get_stats()
        assert (a.conflicts, a.goals, a.timeouts, a.episodes, a.epsilon) == (b.conflicts, b.goals, b.timeouts, b.episodes, b.epsilon)
