"""The engines of the train step at the sizes where their dispatch changes, against the oracle: populations on both sides of every
limit between the ways the arena and gather engines run, and the tile engine (forced by `tile_edge`) on the worlds whose default is
another engine by now."""
import os
import time

import numpy as np
import pytest

from test_gpu_parity import assert_same, lockstep, pair

pytestmark = pytest.mark.gpu
SMS = 148
THREADS = min(8, os.cpu_count() or 1)


def world(pkg, w, h, n, **kw):
    base = dict(start_mode=pkg.START_RANDOM, goal_mode=pkg.GOAL_SEEDED, num_goals=3, obstacle_kind=pkg.OBST_BERNOULLI, obstacle_p=0.15,
                eps_kind=pkg.EPS_FIXED, eps0=0.3, max_steps=11, lr=0.2)
    base.update(kw)
    return pkg.make_config(w, h, n, **base)


LIMITS = [1, 2, 31, 32, 33, 256, 257, 1024, 1025, 4096, 4097, 8193, 16384, 16385, SMS * 512, SMS * 512 + 1, SMS * 1024, SMS * 1024 + 1, 4 * SMS * 1024 + 77, 1300000]


@pytest.mark.parametrize("n", LIMITS)
def test_population_limits(pkg, orc, n):
    """The last population of one way to run the step and the first of the next: one block's shared memory, one cluster, one environment
    per thread of the whole GPU, streamed from shared and from global memory, dealt by cell or not."""
    w, h = (67, 70) if n <= 1024 else (120, 97)
    cfg = world(pkg, w, h, n, env_offset=5)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    lockstep(gpu, cpu, 3, what="n=%d" % n)
    for k in (14, 70) if n < 200000 else (14,):          # many steps per launch: a step cap that everybody reaches together, a second dealing
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "n=%d, many steps per launch" % n)
    sa, sb = gpu.get_stats(), cpu.get_stats()
    assert (sa.conflicts, sa.goals, sa.timeouts, sa.device_error) == (sb.conflicts, sb.goals, sb.timeouts, 0)


@pytest.mark.parametrize("n", [31, 33, 5000, 80000])
def test_crowded_cells_are_counted_alike(pkg, orc, n):
    """Cells with more than 24 environments, whoever applies their updates: the number of such (cell, step) pairs and of the
    environment-steps on them, against a count of the states the oracle went through."""
    cfg = world(pkg, 9, 8, n, num_goals=1, obstacle_p=0.0, max_steps=0, start_mode=pkg.START_CENTRE if n < 32 else pkg.START_RANDOM)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    cells = chained = 0
    for _ in range(12):
        x, y, _t = cpu.get_state()
        c = np.bincount(y * 9 + x)
        cells += int((c > 24).sum()); chained += int(c[c > 24].sum())
        cpu.train_steps(1)
    gpu.train_steps(12)
    s = gpu.get_stats()
    assert (s.long_chains, s.chained) == (cells, chained)
    assert_same(gpu, cpu, "crowded")


@pytest.mark.parametrize("h,n", [(4722, 300), (4723, 300), (13010, 20), (13011, 20), (13011, 1)])
def test_largest_worlds_of_one_block_and_of_one_warp(pkg, orc, h, n):
    cfg = world(pkg, 1, h, n)
    gpu, cpu = pair(pkg, orc, cfg)
    gpu.train_steps(40); cpu.train_steps(40)
    assert_same(gpu, cpu, "1 x %d" % h)


@pytest.mark.parametrize("n,kw", [(1, {}), (29, {}), (29, {"start_mode": 0}), (700, {}), (3000, {}), (90000, {"legacy_clamp": 1}), (400000, {"start_mode": 0}), (2000, {"start_mode": 0, "max_steps": 0})])
def test_common_start_traps_and_episode_epsilon(pkg, orc, n, kw):
    """Everybody on one start cell (whole warps count once), traps, the clamp, and the epsilon that follows the finished episodes."""
    cfg = world(pkg, 91, 93, n, eps_kind=pkg.EPS_MULT_PER_EPISODE, eps0=1.0, eps_decay=0.9, **kw)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    cells = gpu.get_cells()
    for k in np.flatnonzero(cells == 1)[:40]:
        gpu.add_trap(int(k % 91), int(k // 91), -0.3); cpu.add_trap(int(k % 91), int(k // 91), -0.3)
    for k in (1, 2, 40):
        gpu.train_steps(k); cpu.train_steps(k)
        assert gpu.get_stats().epsilon == cpu.get_stats().epsilon
        assert_same(gpu, cpu, "n=%d after +%d" % (n, k))


@pytest.mark.parametrize("edge", [8, 16])
@pytest.mark.parametrize("w,h,n,kw", [(96, 96, 20000, {}), (3, 2, 70000, {}), (500, 490, 60000, {"max_steps": 20}), (24, 17, 3000, {"eps_kind": 2, "eps_decay": 0.97})])
def test_tile_engine_forced(pkg, orc, edge, w, h, n, kw):
    """What the tile engine alone has: region re-sizing, 32-bit counters, mass restarts through the spill list, its epsilon kernel."""
    cfg = world(pkg, w, h, n, num_goals=1, obstacle_p=0.0 if w < 10 else 0.15, tile_edge=edge, rebucket_every=3, **kw)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    for k in (1, 19, 1, 1, 9):
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "edge %d after +%d" % (edge, k))
    a, b = gpu.eval_rollout(60), cpu.eval_rollout(60)    # reads the tiles' move bytes, leaves the regions alone
    assert (a.reached, a.total_steps) == (b.reached, b.total_steps)
    gpu.train_steps(5); cpu.train_steps(5)
    assert_same(gpu, cpu, "edge %d after the rollout" % edge)
    assert gpu.get_stats().device_error == 0


@pytest.mark.parametrize("w,h", [(7, 5), (1024, 1023), (1025, 1024)])
@pytest.mark.parametrize("n", [1, 33, 1024, 1025, 87000, 90001, 300000, 349504, 349505])
def test_update_batch_limits(pkg, orc, w, h, n):
    """update_batch on both sides of its limits -- one block, the mapped stage (of a context without environments, too), the ring; 32-bit and 64-bit sort keys -- and a transition
    out of range anywhere in the batch, which must leave the table as it was."""
    rng = np.random.RandomState(n + w)
    gpu, cpu = pair(pkg, orc, pkg.make_config(w, h, 1 if n <= 300000 else 0, lr=0.3, gamma=0.95, q_init_kind=pkg.QINIT_UNIFORM, q_init_scale=1.0))
    spot = rng.rand(n) < 0.3                             # a third of the batch on few cells
    b = dict(sx=np.where(spot, rng.randint(0, 3, n), rng.randint(0, w, n)), sy=np.where(spot, h - 1, rng.randint(0, h, n)), a=rng.randint(0, 4, n),
             r=rng.choice([-0.01, 1.0, 0.25], n).astype(np.float32), nx=rng.randint(0, w, n), ny=rng.randint(0, h, n), dn=(rng.rand(n) < 0.2).astype(np.uint8))
    for _ in range(2):
        gpu.update_batch(**b)
        assert cpu.update_batch(**b) == 0
        assert np.array_equal(gpu.get_q(), cpu.get_q())
    for name, bad in (("sx", w), ("sy", -1), ("a", 4), ("nx", -1), ("ny", h)):
        wrong = dict(b)
        wrong[name] = b[name].copy()
        wrong[name][rng.randint(0, n)] = bad
        with pytest.raises(pkg.CudarlError):
            gpu.update_batch(**wrong)
    assert np.array_equal(gpu.get_q(), cpu.get_q())
    gpu.update_batch(**b); cpu.update_batch(**b)
    assert np.array_equal(gpu.get_q(), cpu.get_q()) and gpu.get_stats().device_error == 0


@pytest.mark.parametrize("w,h,n,warm", [(63, 65, 700, 300), (64, 64, 5000, 900), (200, 129, 9000, 1500), (1, 300, 40, 50), (700, 650, 1212415, 20), (700, 650, 1212416, 20),
                                        (640, 641, 1300001, 20), (31, 33, 500, 300), (1, 37824, 400, 60), (1, 37825, 400, 60), (1537, 1500, 9000, 300),
                                        (1537, 1500, 1212416, 20)])
@pytest.mark.parametrize("start", [0, 2])
def test_rollout_limits(pkg, orc, w, h, n, warm, start):
    """The folded rollout: grids around the edges of its 32 x 32 and 64 x 64 tiles and
    between the two, one and four environments per thread, caps below, at and beyond the
    lengths of the paths, a common start cell; the table is taken over from the GPU, so that only the rollout is compared."""
    gpu, cpu = pair(pkg, orc, world(pkg, w, h, n, start_mode=start, max_steps=200, eps0=0.2), threads=THREADS)
    gpu.train_steps(warm)
    cpu.set_q(gpu.get_q())
    for cap in (0, 1, 17, 60) if n > 100000 else (0, 1, 17, 64, 5000):
        a, b = gpu.eval_rollout(cap), cpu.eval_rollout(cap)
        assert (a.envs, a.reached, a.total_steps, a.reward_sum) == (b.envs, b.reached, b.total_steps, b.reward_sum), cap


@pytest.mark.parametrize("w,h,n", [(5, 5, 33), (9, 3, 700), (40, 40, 1000), (3000, 2000, 1024), (1, 1, 1024), (1, 1, 1025), (1, 2, 300000), (10, 10, 1 << 20), (64, 64, 200000), (300, 200, 1300), (2000, 1500, 70001)])
def test_update_batch_crowded_cells(pkg, orc, w, h, n):
    """Cells with more transitions than a chain is followed for: none, some and all of the batch, one
    block with its lists or its sort, one to three passes of the sort across blocks."""
    rng = np.random.RandomState(n)
    gpu, cpu = pair(pkg, orc, pkg.make_config(w, h, 1, lr=0.05, gamma=0.95, q_init_kind=pkg.QINIT_UNIFORM, q_init_scale=1.0))
    hot = rng.rand(n) < 0.4
    b = dict(sx=np.where(hot, np.minimum(w - 1, rng.geometric(0.3, n)), rng.randint(0, w, n)), sy=np.where(hot, h // 2, rng.randint(0, h, n)),
             a=rng.randint(0, 4, n), r=rng.choice([-0.01, 1.0, 0.25], n).astype(np.float32), nx=rng.randint(0, w, n), ny=rng.randint(0, h, n),
             dn=(rng.rand(n) < 0.2).astype(np.uint8))
    for _ in range(2):
        gpu.update_batch(**b)
        assert cpu.update_batch(**b) == 0
        assert np.array_equal(gpu.get_q(), cpu.get_q())
    cells = np.bincount(b["sy"] * w + b["sx"])
    if w * h <= 4096:                                    # no two cells share a chain
        assert gpu.get_stats().long_chains == 2 * int((cells > 32).sum())
    assert gpu.get_stats().device_error == 0


@pytest.mark.parametrize("w,h", [(1, 65535 * 64), (1, 65535 * 64 + 1), (1, 65536 * 64 + 65), (2, 65536 * 64 + 1)])
@pytest.mark.parametrize("down", [True, False])
def test_rollout_on_tall_grids(pkg, orc, w, h, down):
    """Grids of more than 65,535 rows of tiles, and the tallest below: everybody walks straight to the goal at one end, through every row of tiles
    on the way, for the whole height and for caps that end some of the walks."""
    cfg = world(pkg, w, h, 20, obstacle_p=0.0, obstacle_kind=pkg.OBST_NONE, goal_mode=pkg.GOAL_LIST, goals=[(x, h - 1 if down else 0) for x in range(w)], num_goals=w)
    gpu, cpu = pair(pkg, orc, cfg)
    q = np.zeros((h, w, 4), np.float32)
    q[..., 2 if down else 0] = 1.0
    gpu.set_q(q); cpu.set_q(q)
    for cap in (h, h // 2, 70):
        a, b = gpu.eval_rollout(cap), cpu.eval_rollout(cap)
        assert (a.envs, a.reached, a.total_steps) == (b.envs, b.reached, b.total_steps), cap
        assert cap < h or a.reached == 20


@pytest.mark.parametrize("n", [20, 2000, 300000])
def test_calls_that_wait_report_a_failure_of_the_device(pkg, n):
    """A wait inside a kernel has run out (the tests' poll bound): every call that hands results back says so, instead of returning what a
    kernel left half done as if it were whole -- update_batch in one block and with its sort, results through the stage and through the ring."""
    g = pkg.VecGridWorld(world(pkg, 90, 80, n))
    g.set_trace(True)
    g.train_steps(1); g.synchronize()
    g.debug_set_copy_wait_polls(1)
    g.train_steps(1)
    g.debug_set_copy_wait_polls(0)
    rng = np.random.RandomState(n)

    def batch(m):
        return dict(sx=np.full(m, 3), sy=np.full(m, 4), a=rng.randint(0, 4, m), r=np.ones(m, np.float32), nx=np.full(m, 3), ny=np.full(m, 5), dn=np.zeros(m, np.uint8))
    calls = dict(update_small=lambda: g.update_batch(**batch(100)), update_sorted=lambda: g.update_batch(**batch(5000)), rollout=lambda: g.eval_rollout(50),
                 step=lambda: g.step_actions(np.zeros(n, np.int32)), reward_done=g.get_reward_done, trace=g.get_trace, state=g.get_state, q=g.get_q,
                 synchronize=g.synchronize, stats=g.get_stats)
    for name, call in calls.items():
        with pytest.raises(pkg.CudarlError) as ei:
            call()
            pytest.fail(name)
        assert ei.value.code == 3000 + 32, name


@pytest.mark.parametrize("n", [5000, 16384, 60000, SMS * 512, 90000, 4 * SMS * 1024 + 77])
def test_episode_epsilon_when_everybody_ends_in_the_first_step_of_a_launch(pkg, orc, n):
    """The epsilon of a step follows the episodes finished before it.  All environments reach the step cap in the first step of a launch of many:
    no block may see the episodes of that step when it looks up the epsilon it begins with.  One cluster, the whole GPU, dealt by cell or not."""
    cfg = world(pkg, 120, 97, n, num_goals=1, max_steps=8, eps_kind=pkg.EPS_MULT_PER_EPISODE, eps0=1.0, eps_decay=0.6)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    for k in (7, 8, 8, 8, 8, 8, 64) if n < 100000 else (7, 8, 8):
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "n=%d after +%d" % (n, k))
        assert gpu.get_stats().epsilon == cpu.get_stats().epsilon


@pytest.mark.parametrize("n", [0, 1, 32])
def test_memory_of_contexts_that_need_no_counters(pkg, n):
    """A table with no or few environments: 16 bytes a cell, 4 for the rollout, 2 for the cell's class and 1 for its moves."""
    import torch
    side = 6000
    pkg.VecGridWorld(world(pkg, 8, 8, 1)).close()            # what the process needs once
    free = torch.cuda.mem_get_info()[0]
    w = pkg.VecGridWorld(world(pkg, side, side, n))
    used = free - torch.cuda.mem_get_info()[0]
    assert used < 23 * side * side + (32 << 20)
    w.train_steps(3); w.eval_rollout(5); w.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 23 * side * side + (32 << 20)


@pytest.mark.parametrize("n,lr", [(90000, 0.001), (400000, 1e-4), (1 << 20, 1e-5)])
def test_a_crowd_of_slow_learners(pkg, orc, n, lr):
    """Everybody on one start cell, and updates that are far from their fixed point after as many rounds as there are environments: one of them makes
    the rounds for all.  When each made them for itself, 16 steps of the largest crowd took 1.7 s; they take less than a tenth of that."""
    cfg = world(pkg, 301, 299, n, start_mode=pkg.START_CENTRE, lr=lr, eps0=0.1, max_steps=0)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    gpu.synchronize()
    t = time.perf_counter()
    gpu.train_steps(16); gpu.synchronize()
    t = time.perf_counter() - t
    cpu.train_steps(16)
    assert_same(gpu, cpu, "n=%d lr=%g" % (n, lr))
    assert t < 0.8


def test_one_step_a_call_does_not_deal_every_step(pkg, orc):
    """Dealt by cell every 64 steps, however many calls those are (a dealing in every launch took 13 us a step on top of the step's 7, a launch
    alone takes 5); calls of any length in a row, and with the records read and replaced between them, leave the same world."""
    cfg = world(pkg, 300, 290, 100000, max_steps=150)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    for k in (1, 1, 61, 1, 1, 64, 65, 3, 127, 1):
        gpu.train_steps(k); cpu.train_steps(k)
        if k in (61, 65, 3):
            assert_same(gpu, cpu, "+%d" % k)
        if k == 64:
            x, y, t = gpu.get_state()
            gpu.set_state(t=t); cpu.set_state(t=t)       # back to the order of the environments
    assert_same(gpu, cpu, "after all")

    def best(calls, steps):
        times = []
        for _ in range(15):
            gpu.synchronize()
            t = time.perf_counter()
            for _ in range(calls):
                gpu.train_steps(steps)
            gpu.synchronize()
            times.append(time.perf_counter() - t)
        return min(times)
    assert best(64, 1) < best(1, 64) + 64 * 9e-6


@pytest.mark.parametrize("n", [1, 300, 21800, 349504, 349505, 1 << 20])
def test_set_state_limits(pkg, n):
    """States in through the mapped stage and through the ring, all or some of the arrays, and one value out of range anywhere, which must leave the
    states as they were.  (Checked by one core before it was copied, the largest took 2.2 ms.)"""
    g = pkg.VecGridWorld(world(pkg, 1000, 777, n, obstacle_p=0.0, obstacle_kind=pkg.OBST_NONE, max_steps=0))
    g.train_steps(2)
    rng = np.random.RandomState(n)
    x, y, t = rng.randint(0, 1000, n).astype(np.int32), rng.randint(0, 777, n).astype(np.int32), rng.randint(0, 0xFFFFFE + 1, n).astype(np.int32)
    g.set_state(x, y, t)
    assert all(np.array_equal(a, b) for a, b in zip(g.get_state(), (x, y, t)))
    for k, bad in ((0, 1000), (0, -1), (1, 777), (1, -5), (2, 0xFFFFFF), (2, -1)):
        wrong = [x.copy(), y.copy(), t.copy()]
        wrong[k][rng.randint(0, n)] = bad
        with pytest.raises(pkg.CudarlError) as ei:
            g.set_state(*wrong)
        assert ei.value.code == -3 and ("step count" in str(ei.value)) == (k == 2)
    assert all(np.array_equal(a, b) for a, b in zip(g.get_state(), (x, y, t)))
    y = y[::-1].copy()
    g.set_state(y=y)
    assert all(np.array_equal(a, b) for a, b in zip(g.get_state(), (x, y, t)))
    times = []
    for _ in range(15):
        s = time.perf_counter()
        g.set_state(x, y, t)
        times.append(time.perf_counter() - s)
    assert min(times) < 1.2e-3
