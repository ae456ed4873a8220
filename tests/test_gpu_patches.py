"""The patch engine of the train step against the oracle: launches of many steps of worlds cut into patches of every shape, the ways out of it in the
middle of a launch -- a patch with more environments than slots, more records in a step than the receiver has room for -- and when it is not taken: crowded grids, few
goals, other contexts' steps under way, no memory."""
import ctypes as C
import os
import threading

import numpy as np
import pytest

from test_gpu_engines import world
from test_gpu_parity import assert_same, pair

pytestmark = pytest.mark.gpu
THREADS = min(8, os.cpu_count() or 1)


def same_stats(gpu, cpu):
    a, b = gpu.get_stats(), cpu.get_stats()
    assert (a.conflicts, a.goals, a.timeouts, a.episodes, a.epsilon, a.device_error) == (b.conflicts, b.goals, b.timeouts, b.episodes, b.epsilon, 0)


@pytest.mark.parametrize("w,h,n", [
    (40, 30, 1100), (64, 64, 4096), (120, 97, 1025),
    (97, 120, 2048), (97, 120, 2049), (97, 120, 4096), (97, 120, 4097), (97, 120, 8192), (97, 120, 8193), (97, 120, 10240), (97, 120, 10241),       # both sides of 256 and 512 threads; the most environments
    (160, 161, 12288), (160, 161, 12289),
    (5000, 1, 33), (1, 5000, 1025), (7, 3000, 6000), (3000, 9, 6000),        # one cell wide, one high: most of a band is empty
    (3, 2, 5000), (2, 1, 1500),  # fewer bins of cells than blocks: patches without a cell
    (340, 330, 1500),            # the map of start cells does not fit
    # on all multiprocessors: both sides of 512 threads, the most environments, the most for three goals; a large grid; one that does not fit
    (420, 400, 1500), (9000, 3, 20000), (130, 110, 37888), (256, 256, 37889), (256, 256, 65536), (400, 300, 113664), (400, 300, 113665), (256, 256, 88680), (256, 256, 88682),
    (1001, 613, 70001), (1300, 1100, 2000), (1000, 900, 20000), (1100, 1024, 3000),      # the third from last does not fit, the others nearly fill the shared memory
])
def test_worlds_cut_into_patches(pkg, orc, w, h, n):
    cfg = world(pkg, w, h, n, num_goals=1 if w * h < 100 else 3, obstacle_p=0.0 if w * h < 100 else 0.15, max_steps=37, env_offset=3)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    for k in (15, 16, 2, 31, 32, 90) + ((127, 128) if n > 37888 else ()) + ((w * h // 8192 + 1,) if w * h > 1 << 18 else ()):        # one less than the fewest steps of such a launch, the fewest, a launch of the other engine between
        gpu.set_trace(k != 90)                       # with and without the options
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "+%d" % k)
        assert k == 90 or all(np.array_equal(a, b) for a, b in zip(gpu.get_trace(), cpu.get_trace()))
    same_stats(gpu, cpu)


@pytest.mark.parametrize("w,h,n,patches", [
    (32, 32, 4096, True), (32, 32, 4097, False), (16, 16, 1025, False), (64, 64, 8192, True), (64, 64, 8193, False), (97, 120, 8193, True), (70, 73, 10220, True), (70, 73, 10221, False)])
def test_crowded_grids_are_not_cut(pkg, orc, w, h, n, patches):
    """Both sides of the limits of environments a cell, and of the most in a cluster."""
    gpu, cpu = pair(pkg, orc, world(pkg, w, h, n, max_steps=37), threads=THREADS)
    if n > 8192:
        assert makes_buffers(gpu, 40) == patches
    else:
        gpu.train_steps(20); gpu.train_steps(40)
    cpu.train_steps(60)
    for k in (15, 16, 31, 32, 90):
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "+%d" % k)
    same_stats(gpu, cpu)


@pytest.mark.parametrize("w,h,n", [(91, 93, 3000), (201, 199, 8000), (301, 299, 80000)])
@pytest.mark.parametrize("kw", [{"eps_kind": 2, "eps0": 1.0, "eps_decay": 0.9}, {"eps_kind": 1, "eps0": 1.0, "eps_decay": 0.99},
                                {"eps_kind": 3, "eps0": 1.0, "eps_end": 0.1, "eps_steps": 60, "legacy_clamp": 1}])
def test_epsilons_traps_and_clamp(pkg, orc, w, h, n, kw):
    """The epsilon of a step that follows the episodes all blocks have finished before it; by step, in launches that start anywhere in its table."""
    cfg = world(pkg, w, h, n, **kw)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    cells = gpu.get_cells()
    for k in np.flatnonzero(cells == 1)[:60]:
        gpu.add_trap(int(k % w), int(k // w), -0.3); cpu.add_trap(int(k % w), int(k // w), -0.3)
    for k in (16, 1, 33, 47) + ((129, 131) if n > 37888 else ()):
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "+%d" % k)
        same_stats(gpu, cpu)


def crowd_world(pkg, n, **kw):
    return world(pkg, 200, 190, n, num_goals=1, obstacle_p=0.0, obstacle_kind=pkg.OBST_NONE, goal_mode=pkg.GOAL_LIST, goals=[(199, 189)], **kw)


@pytest.mark.parametrize("n", [3000, 12000, 38000])
@pytest.mark.parametrize("together", [False, True])
def test_crowds_that_no_patch_holds(pkg, orc, n, together):
    """Everybody on one cell when a launch begins, or -- the rows lead all of them there -- by its middle; spread out again later."""
    cfg = crowd_world(pkg, n, max_steps=90, eps0=0.02, lr=0.05)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    y, x = np.mgrid[0:190, 0:200]
    q = np.zeros((190, 200, 4), np.float32)
    q[..., 1] = x < 100; q[..., 3] = x > 100             # towards the middle column, along it towards the middle
    q[..., 2] = (x == 100) & (y < 95); q[..., 0] = (x == 100) & (y >= 95)
    gpu.set_q(q); cpu.set_q(q)
    if together:
        for m in (gpu, cpu):
            m.set_state(np.full(n, 20, np.int32), np.full(n, 30, np.int32), None)
    for k in (16, 150, 30):
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "+%d" % k)
        same_stats(gpu, cpu)


@pytest.mark.parametrize("w,h,n", [(200, 190, 3000), (200, 190, 38000), (400, 390, 90000)])
@pytest.mark.parametrize("kw", [{}, {"eps_kind": 2, "eps0": 0.2, "eps_decay": 0.9}])
def test_patches_given_up_are_tried_again_later(pkg, orc, w, h, n, kw):
    """A crowd that no patch holds for hundreds of steps, in short calls with others of the gather engine between (it deals 90,000 environments by cell); then everybody begins anew."""
    cfg = world(pkg, w, h, n, num_goals=2, obstacle_p=0.0, obstacle_kind=pkg.OBST_NONE, goal_mode=pkg.GOAL_LIST, goals=[(w - 1, h - 1), (0, h - 1)], **dict(dict(max_steps=150, eps0=0.02, lr=0.05), **kw))
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    rng = np.random.RandomState(n)
    crowd = np.where(rng.rand(n) < 0.97, 20, rng.randint(0, w, n)).astype(np.int32)
    for turn in range(3):
        for m in (gpu, cpu):
            m.set_state(crowd, np.full(n, 30, np.int32), None)
        for k in (33, 64, 5, 40):
            gpu.train_steps(k); cpu.train_steps(k)
            assert_same(gpu, cpu, "turn %d, +%d" % (turn, k))
        for m in (gpu, cpu):
            m.reset_all()
        for k in (200, 7, 300):
            gpu.train_steps(k); cpu.train_steps(k)
            assert_same(gpu, cpu, "turn %d, again, +%d" % (turn, k))
            same_stats(gpu, cpu)


@pytest.mark.parametrize("n", [2500, 10000, 38000])
def test_many_cross_at_once(pkg, orc, n):
    """All environments of a few cells walk abreast: more records in a step than their receiver has room for."""
    cfg = crowd_world(pkg, n, max_steps=0, eps0=0.0, lr=0.001)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    rng = np.random.RandomState(n)
    q = np.zeros((190, 200, 4), np.float32); q[..., 1] = 1000.0
    x, y = rng.randint(0, 8, n).astype(np.int32), (rng.randint(0, 3, n) * 60).astype(np.int32)
    for m in (gpu, cpu):
        m.set_q(q); m.set_state(x, y, np.zeros(n, np.int32))
    for k in (16, 100, 40):
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "+%d" % k)
    same_stats(gpu, cpu)


@pytest.mark.parametrize("w,h,n,rows,each", [(400, 400, 16000, 32, 400), (200, 190, 2500, 64, 250)])
def test_a_column_walks_abreast(pkg, orc, w, h, n, rows, each):
    """`each` environments on every eight cells of a column, few enough for the patches there, all of which step into the wide patch beside them at once: more than its list
    of arrivals holds -- on the whole GPU, and in a cluster."""
    cfg = world(pkg, w, h, n, num_goals=1, obstacle_p=0.0, obstacle_kind=pkg.OBST_NONE, goal_mode=pkg.GOAL_LIST, goals=[(w - 1, h - 1)], max_steps=0, eps0=0.0, lr=0.001)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    rng = np.random.RandomState(n)
    q = np.zeros((h, w, 4), np.float32); q[..., 1] = 1000.0
    m = each * rows // 8
    for at in (5, 40):
        x, y = rng.randint(at + 1, w, n).astype(np.int32), rng.randint(0, h, n).astype(np.int32)
        x[:m] = at; y[:m] = np.arange(m) % rows
        for k in (gpu, cpu):
            k.set_q(q); k.set_state(x, y, np.zeros(n, np.int32))
        for k in (64, 100):
            gpu.train_steps(k); cpu.train_steps(k)
            assert_same(gpu, cpu, "+%d" % k)
    same_stats(gpu, cpu)


def counted_crowds(cpu, w, steps):
    """Trains the oracle; (cell, step) pairs with more than 24 environments, and the environments on them."""
    cells = chained = 0
    for _ in range(steps):
        x, y, _t = cpu.get_state()
        c = np.bincount(y * w + x)
        cells += int((c > 24).sum()); chained += int(c[c > 24].sum())
        cpu.train_steps(1)
    return cells, chained


@pytest.mark.parametrize("w,h,n,k", [(60, 60, 1500, 40), (60, 60, 3000, 40), (80, 80, 8000, 40), (120, 120, 20000, 64), (300, 290, 40000, 140)])
@pytest.mark.parametrize("together", [False, True])
def test_crowded_cells_of_patches(pkg, orc, w, h, n, k, together):
    """Cells with more than 24 environments, in patches to the end and in patches that are given up when the rows have led everybody to one place."""
    cfg = world(pkg, w, h, n, num_goals=2, obstacle_p=0.0, obstacle_kind=pkg.OBST_NONE, goal_mode=pkg.GOAL_LIST, goals=[(w - 1, h - 1), (0, h - 1)], max_steps=200, eps0=0.05)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    rng = np.random.RandomState(n)
    x, y = rng.randint(0, w, n).astype(np.int32), rng.randint(0, h, n).astype(np.int32)
    crowd = rng.randint(0, 2 * n, n)                     # eight cells with a fortieth of the population each, or some 375
    m = (crowd < 100 * min(n // 100, 150)) & (crowd % 100 < 40)
    x[m], y[m] = (crowd[m] % 4) * (w // 4), (crowd[m] // 4 % 2) * (h // 2)
    if together:
        my, mx = np.mgrid[0:h, 0:w]
        q = np.zeros((h, w, 4), np.float32); cx, cy = w // 2, h // 2
        q[..., 1] = mx < cx; q[..., 3] = mx > cx; q[..., 2] = (mx == cx) & (my < cy); q[..., 0] = (mx == cx) & (my >= cy)
        gpu.set_q(q); cpu.set_q(q)
    for v in (gpu, cpu):
        v.set_state(x, y, None)
    cells = chained = 0
    for steps in (k, 2 * k):
        more = counted_crowds(cpu, w, steps)
        gpu.train_steps(steps)
        cells += more[0]; chained += more[1]
        s = gpu.get_stats()
        assert (s.long_chains, s.chained) == (cells, chained)
        assert_same(gpu, cpu, "+%d" % steps)
    assert cells > 0
    same_stats(gpu, cpu)


@pytest.mark.parametrize("n", [3000, 8000, 20000, 38000])
@pytest.mark.parametrize("kw", [{"eps_kind": 1, "eps0": 0.3, "eps_decay": 0.98}, {"eps_kind": 2, "eps0": 0.3, "eps_decay": 0.9}, {"eps_kind": 3, "eps0": 0.3, "eps_end": 0.02, "eps_steps": 150, "legacy_clamp": 1}])
def test_patches_given_up_with_options(pkg, orc, n, kw):
    """Patches that a crowd ends in the middle of a launch: the epsilon goes on where it was, by step and by the episodes of all blocks, with traps, a trace and the clamp."""
    w, h = 200, 190
    cfg = world(pkg, w, h, n, num_goals=2, obstacle_p=0.02, goal_mode=pkg.GOAL_LIST, goals=[(100, 94), (199, 189)], max_steps=70, lr=0.05, **kw)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    for c in np.flatnonzero(gpu.get_cells() == 1)[:200]:
        gpu.add_trap(int(c % w), int(c // w), -0.3); cpu.add_trap(int(c % w), int(c // w), -0.3)
    y, x = np.mgrid[0:h, 0:w]
    q = np.zeros((h, w, 4), np.float32)
    q[..., 1] = x < 100; q[..., 3] = x > 100; q[..., 2] = (x == 100) & (y < 94); q[..., 0] = (x == 100) & (y > 94)
    gpu.set_q(q); cpu.set_q(q)
    gpu.set_trace(True)
    for k in (130, 33, 200):
        gpu.train_steps(k); cpu.train_steps(k)
        assert_same(gpu, cpu, "+%d" % k)
        assert all(np.array_equal(a, b) for a, b in zip(gpu.get_trace(), cpu.get_trace()))
        same_stats(gpu, cpu)


@pytest.mark.parametrize("w,h,n", [(9, 8, 20), (20, 19, 300), (32, 32, 1000), (64, 64, 1500), (64, 64, 4096), (90, 93, 8000), (120, 120, 20000), (300, 290, 40000)])
@pytest.mark.parametrize("seed", range(2))
def test_rows_with_ties_infinities_and_no_numbers(pkg, orc, w, h, n, seed):
    """In worlds of one block, in clusters and on the whole GPU: rows, edge values and counted updates."""
    rng = np.random.RandomState(seed)
    gpu, cpu = pair(pkg, orc, world(pkg, w, h, n, num_goals=1 if n < 38000 else 8, obstacle_p=0.1, max_steps=13, eps0=0.2, lr=0.5, legacy_clamp=seed), threads=THREADS)
    q = rng.choice(np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, np.nan, -3.4e38, 1e-42], np.float32), (h, w, 4))
    gpu.set_q(q); cpu.set_q(q)
    for k in (1, 40, 130):
        gpu.train_steps(k); cpu.train_steps(k)
        assert all(np.array_equal(a, b) for a, b in zip(gpu.get_state(), cpu.get_state())), "+%d" % k
        assert np.array_equal(gpu.get_q(), cpu.get_q(), equal_nan=True), "+%d" % k
        same_stats(gpu, cpu)


@pytest.mark.parametrize("n", [9000, 30000])
def test_table_and_states_changed_between_launches(pkg, orc, n):
    """Nothing of a launch is left in the next: the table set and updated, states set, cells changed in between."""
    cfg = world(pkg, 150, 140, n, max_steps=60)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    rng = np.random.RandomState(5)
    for turn in range(4):
        gpu.train_steps(16); cpu.train_steps(16)
        assert_same(gpu, cpu, "turn %d" % turn)
        q = rng.uniform(0, 1, (140, 150, 4)).astype(np.float32)
        x, y = rng.randint(0, 150, n).astype(np.int32), rng.randint(0, 140, n).astype(np.int32)
        b = dict(sx=rng.randint(0, 150, 2000), sy=rng.randint(0, 140, 2000), a=rng.randint(0, 4, 2000), r=np.ones(2000, np.float32),
                 nx=rng.randint(0, 150, 2000), ny=rng.randint(0, 140, 2000), dn=np.zeros(2000, np.uint8))
        for m in (gpu, cpu):
            m.set_q(q); m.set_state(x, y, None); m.update_batch(**b); m.add_obstacle(3 + turn, 4); m.set_goal(100 + turn, 20)
    gpu.train_steps(30); cpu.train_steps(30)
    assert_same(gpu, cpu, "last")
    same_stats(gpu, cpu)


@pytest.mark.parametrize("n", [5000, 30000])
def test_a_failed_wait_ends_the_launch(pkg, n):
    """With the tests' poll bound a launch records the failure and leaves; every later launch does nothing."""
    g = pkg.VecGridWorld(world(pkg, 120, 97, n))
    g.train_steps(20); g.synchronize()
    g.debug_set_copy_wait_polls(1)
    g.train_steps(20)
    g.debug_set_copy_wait_polls(0)
    g.train_steps(20)
    with pytest.raises(pkg.CudarlError) as ei:
        g.synchronize()
    assert ei.value.code == 3000 + 32


def test_buffers_that_cannot_be_had(pkg, orc):
    """The patches' buffers (here 20 MB) are made by the first launch of them: where there is no memory left, the steps run as they do without."""
    gpu, cpu = pair(pkg, orc, world(pkg, 1000, 900, 20000, eps_kind=pkg.EPS_MULT_PER_STEP, eps0=1.0, eps_decay=0.99), threads=THREADS)
    gpu.train_steps(20); cpu.train_steps(20)
    assert_same(gpu, cpu, "before")
    rt = _runtime()
    held, size = [], 1 << 36
    while size >= 1 << 23:
        p = C.c_void_p()
        if rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0:
            held.append(p)
        else:
            size //= 2
    try:
        gpu.train_steps(150)
        gpu.synchronize()
    finally:
        rt.cudaGetLastError()
        for p in held:
            rt.cudaFree(p)
    cpu.train_steps(150)
    gpu.train_steps(150); cpu.train_steps(150)
    assert_same(gpu, cpu, "after")
    same_stats(gpu, cpu)


def makes_buffers(gpu, n):
    """Whether training n steps makes the patches' buffers, as the first launch of patches does (on the whole GPU more than 4 MB)."""
    free, total = C.c_size_t(), C.c_size_t()
    left = []
    for k in (20, n):
        gpu.train_steps(k); gpu.synchronize()
        assert _runtime().cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
        left.append(free.value)
    return left[0] - left[1] >= 4 << 20


def test_engine_follows_the_goals(pkg, orc):
    """65,536 environments on 256 x 256 cells take patches with eight goals, not with one; set_goal leaves one."""
    cfg = world(pkg, 256, 256, 65536, num_goals=8)
    other = pkg.VecGridWorld(cfg)
    assert not makes_buffers(other, 107) and makes_buffers(other, 128) and not makes_buffers(other, 128)
    gpu, cpu = pair(pkg, orc, cfg, threads=THREADS)
    gpu.set_goal(100, 100)
    assert not makes_buffers(gpu, 600)
    cpu.set_goal(100, 100); cpu.train_steps(620)
    assert_same(gpu, cpu, "one goal")


def test_room_beside_other_worlds(pkg, orc):
    """A launch on the whole GPU would wait for the steps of another context, and its steps for the launch: while they are under way, the gather engine takes them."""
    other = pkg.VecGridWorld(world(pkg, 120, 97, 5000))
    other.train_steps(64); other.synchronize()
    gpu, cpu = pair(pkg, orc, world(pkg, 350, 350, 3000), threads=THREADS)
    other.train_steps(150000)                            # some 0.4 s
    assert not makes_buffers(gpu, 200)
    other.synchronize()
    assert makes_buffers(gpu, 200)
    cpu.train_steps(440)
    assert_same(gpu, cpu, "beside another")
    same_stats(gpu, cpu)


def test_many_worlds_at_once(pkg, orc):
    """More worlds than there is room for as clusters, each trained by a thread of its own, some on the whole GPU, some let go while others train."""
    sizes = [(50, 50, 1500), (64, 64, 4096), (350, 350, 3000), (20, 20, 200)] * 3
    wrong = []

    def one(k, w, h, n):
        try:
            for again in range(2):
                cfg = world(pkg, w, h, n, seed=k + 100 * again)
                gpu, cpu = pair(pkg, orc, cfg)
                for m in (64, 33, 200, 16):
                    gpu.train_steps(m); cpu.train_steps(m)
                gpu.train_steps(40); cpu.train_steps(40)
                assert_same(gpu, cpu, "world %d" % k)
                gpu.close()
        except Exception as e:
            wrong.append(e)
    threads = [threading.Thread(target=one, args=(k,) + s) for k, s in enumerate(sizes)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def _runtime():
    return next(lib for lib in map(_library, ("libcudart.so.12", "libcudart.so", "/usr/local/cuda/lib64/libcudart.so.12")) if lib)


def _library(name):
    try:
        return C.CDLL(name)
    except OSError:
        return None
