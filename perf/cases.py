"""Performance cases: what a user of this framework has it do, through its public entry points.

A case is a dict of plain values.  `prepare` builds what the user's program has in hand before the call (a world in the middle
of its training run, a batch of transitions, an array of actions), `run` makes one pass, `work` states the bytes and operations
the pass cannot do without.  Five kinds of use:

  train   n fused steps of all environments (epsilon-greedy, move, TD update, auto-reset), then the table, the environments'
          states and the run statistics are read back -- a training program between two checkpoints;
  eval    one greedy rollout of every environment on the table as it stands;
  update  mini-batches of recorded transitions through the ordered TD update, then the table is read back -- learning from a
          replay buffer;
  step    one step of all environments with the caller's actions, rewards, done flags and positions back on the host -- a policy
          of the user's own drives the environments;
  env     one episode of a single `cudarl_core.Environment`, step by step from Python -- the loop of a reference-style agent.

Everything here is deterministic: states, actions, counters and the fp32 table have to come out the same to the last bit, because
one differing bit of the table changes an argmax and the trajectories part.
"""
import importlib.util
import math
import os
import sys

import numpy as np


def _package():
    name = "cudarl_arena_b200"
    if name not in sys.modules:
        here = os.path.join(os.getcwd(), "cudarl-arena_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(here, "__init__.py"), submodule_search_locations=[here])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


def _core():
    here = os.path.join(os.getcwd(), "cudarl-arena_b200")
    if here not in sys.path:
        sys.path.append(here)
    import cudarl_core
    return cudarl_core


def listed():
    return [
        # The reference's own use: a Python agent steps one 10 x 10 environment through the pybind module.
        dict(name="env_10x10", kind="env", width=10, height=10, steps=200),
        # The reference's default training configuration: one environment, one episode's cap of steps.  Launch latency.
        dict(name="train_10x10_1", kind="train", width=10, height=10, envs=1, steps=500, warm=1000, obstacles="bernoulli", p=0.1,
             goals=1, cap=500, lr=0.1, gamma=0.99, eps="episode", clamp=False, traps=0),
        # A small arena once the policy has formed: thousands of environments on the same few paths to the only goal.
        dict(name="train_64x64_4k", kind="train", width=64, height=64, envs=4096, steps=1024, warm=6144, obstacles="bernoulli",
             p=0.15, goals=1, cap=1024, lr=0.1, gamma=0.99, eps="fixed", clamp=False, traps=0),
        # A medium arena with a decaying epsilon, well into its training run.
        dict(name="train_256x256_64k", kind="train", width=256, height=256, envs=65536, steps=512, warm=12288, obstacles="bernoulli",
             p=0.2, goals=8, cap=4096, lr=0.05, gamma=0.99, eps="linear", clamp=False, traps=0),
        # A maze of walls, as many environments as cells.
        dict(name="train_1024x1024_1m", kind="train", width=1024, height=1024, envs=1 << 20, steps=256, warm=512, obstacles="walls",
             p=0.25, goals=1, cap=4096, lr=0.1, gamma=0.995, eps="fixed", clamp=False, traps=0),
        # The headline configuration: a table larger than L2, 4.2 million environments.
        dict(name="train_4096x4096_4m", kind="train", width=4096, height=4096, envs=1 << 22, steps=1024, warm=256,
             obstacles="bernoulli", p=0.3, goals=64, cap=16384, lr=0.1, gamma=0.99, eps="fixed", clamp=False, traps=0),
        # Nothing is a power of two: ragged grid, traps, the flat reference kernel's clamp, epsilons from the host for every call.
        dict(name="train_1001x613_150k", kind="train", width=1001, height=613, envs=150001, steps=300, warm=600, obstacles="walls",
             p=0.2, goals=5, cap=777, lr=0.1, gamma=0.98, eps="host", clamp=True, traps=99),
        # Evaluation between training phases: a formed policy on the medium arena, an early one on the headline arena.
        dict(name="eval_256x256_64k", kind="eval", width=256, height=256, envs=65536, steps=1000, warm=12288, obstacles="bernoulli",
             p=0.2, goals=8, cap=4096, lr=0.05, gamma=0.99, eps="linear", clamp=False, traps=0),
        dict(name="eval_4096x4096_4m", kind="eval", width=4096, height=4096, envs=1 << 22, steps=1000, warm=1024,
             obstacles="bernoulli", p=0.3, goals=64, cap=16384, lr=0.1, gamma=0.99, eps="fixed", clamp=False, traps=0),
        # Replay mini-batches of the size the reference's update_batch takes, and one of a million odd transitions.
        dict(name="update_64x64_1k", kind="update", width=64, height=64, batch=1000, calls=16, hot=0.5, lr=0.1, gamma=0.99, clamp=False),
        dict(name="update_1024x1024_1m", kind="update", width=1024, height=1024, batch=1000003, calls=4, hot=0.5, lr=0.1, gamma=0.99,
             clamp=False),
        # The caller's own policy drives 65,536 environments.
        dict(name="step_256x256_64k", kind="step", width=256, height=256, envs=65536, p=0.2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "eval", "update", "step", "env"])
    side = _log(rng, 10, 4096)
    w = side
    h = max(10, min(4096, _log(rng, side / 2, side * 2)))
    cells = w * h
    if kind == "env":
        return dict(kind="env", width=rng.randint(5, 40), height=rng.randint(5, 40), steps=rng.randint(50, 300))
    if kind == "update":
        return dict(kind="update", width=w, height=h, batch=_log(rng, 16, 1 << 20), calls=rng.randint(2, 8), hot=rng.choice([0.0, 0.5]),
                    lr=rng.choice([0.05, 0.1]), gamma=rng.choice([0.98, 0.99]), clamp=rng.random() < 0.25)
    envs = max(1, min(1 << 22, int(cells * math.exp(rng.uniform(math.log(1 / 64), math.log(1.5))))))
    if kind == "step":
        return dict(kind="step", width=w, height=h, envs=envs, p=rng.choice([0.0, 0.1, 0.2, 0.3]))
    case = dict(kind=kind, width=w, height=h, envs=envs, obstacles=rng.choice(["none", "bernoulli", "walls"]), p=rng.choice([0.1, 0.15, 0.2, 0.25]),
                goals=rng.choice([1, 1, 5, 8, 64]) if cells > 1000 else 1, cap=_log(rng, 200, 16384), lr=rng.choice([0.05, 0.1]),
                gamma=rng.choice([0.98, 0.99, 0.995]), eps=rng.choice(["fixed", "fixed", "linear", "step", "episode", "host"]),
                clamp=rng.random() < 0.1, traps=rng.choice([0, 0, 0, 20]))
    spread = 1 + envs // 40000                       # a batched step of this many environments costs about that many times a small one
    case["warm"] = max(64, 6000 // spread)
    case["steps"] = _log(rng, 100, 2000) if kind == "eval" else max(32, _log(rng, 200, 1500) // (1 + spread // 16))
    return case


def _world(case, seed):
    """The world of a train / eval case, `warm` steps into its training run."""
    pkg = _package()
    obst = {"none": pkg.OBST_NONE, "bernoulli": pkg.OBST_BERNOULLI, "walls": pkg.OBST_WALLS}[case["obstacles"]]
    eps = {"fixed": dict(eps_kind=pkg.EPS_FIXED, eps0=0.1), "host": dict(eps_kind=pkg.EPS_FIXED, eps0=0.1),
           "linear": dict(eps_kind=pkg.EPS_LINEAR, eps0=1.0, eps_end=0.05, eps_steps=100000),
           "step": dict(eps_kind=pkg.EPS_MULT_PER_STEP, eps0=1.0, eps_decay=0.9995),
           "episode": dict(eps_kind=pkg.EPS_MULT_PER_EPISODE, eps0=1.0, eps_decay=0.995)}[case["eps"]]
    one = case["envs"] == 1
    start = dict(start_mode=pkg.START_FIXED, start_x=0, start_y=0, goals=[(case["width"] - 1, case["height"] - 1)]) if one else \
        dict(start_mode=pkg.START_RANDOM, goal_mode=pkg.GOAL_SEEDED, num_goals=case["goals"])
    world = pkg.VecGridWorld(pkg.make_config(case["width"], case["height"], case["envs"], 0xC0DA2025 + seed, obstacle_kind=obst,
                                             obstacle_p=case["p"], max_steps=case["cap"], lr=case["lr"], gamma=case["gamma"],
                                             legacy_clamp=int(case["clamp"]), q_init_kind=pkg.QINIT_UNIFORM, q_init_scale=0.01, **start, **eps))
    rng = np.random.default_rng(seed)
    if case["traps"]:
        for cell in rng.choice(np.flatnonzero(world.get_cells() == 1), case["traps"]) if (world.get_cells() == 1).any() else []:
            world.add_trap(int(cell % case["width"]), int(cell // case["width"]), -0.25)
    world.train_steps(case["warm"])
    world.synchronize()
    return world


def _batch(case, rng):
    """Recorded transitions: uniform over the grid, a part of them around one busy place, neighbours as next cells."""
    n, w, h = case["batch"], case["width"], case["height"]
    x, y = rng.integers(0, w, n), rng.integers(0, h, n)
    hot = rng.random(n) < case["hot"]
    x = np.where(hot, np.clip(rng.normal(w / 2, w / 8, n).astype(np.int64), 0, w - 1), x)
    y = np.where(hot, np.clip(rng.normal(h / 2, h / 8, n).astype(np.int64), 0, h - 1), y)
    a = rng.integers(0, 4, n)
    nx = np.clip(x + (a == 1) - (a == 3), 0, w - 1)
    ny = np.clip(y + (a == 2) - (a == 0), 0, h - 1)
    done = rng.random(n) < 0.01
    return [x.astype(np.int32), y.astype(np.int32), a.astype(np.int32), np.where(done, 1.0, -0.01).astype(np.float32), nx.astype(np.int32),
            ny.astype(np.int32), done.astype(np.uint8)]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    state = dict(case=case)
    if case["kind"] == "env":
        env = _core().Environment(case["width"], case["height"], seed & 0xFFFF)
        for cell in rng.integers(0, case["width"] * case["height"], 8):            # a few walls and the goal of the user's own task
            env.add_obstacle(int(cell % case["width"]), int(cell // case["width"]))
        env.set_goal(case["width"] - 1, case["height"] - 1)
        state.update(env=env, actions=rng.integers(0, 4, case["steps"]).tolist())
    elif case["kind"] in ("train", "eval"):
        state["world"] = _world(case, seed)
        if case["eps"] == "host":
            state["eps"] = np.linspace(0.5, 0.05, case["steps"]).astype(np.float32)
    elif case["kind"] == "update":
        pkg = _package()
        state["world"] = pkg.VecGridWorld(pkg.make_config(case["width"], case["height"], 0, 0xC0DA2025 + seed, lr=case["lr"], gamma=case["gamma"],
                                                          legacy_clamp=int(case["clamp"]), q_init_kind=pkg.QINIT_UNIFORM, q_init_scale=0.01))
        state["batches"] = [_batch(case, rng) for _ in range(case["calls"])]
    else:
        pkg = _package()
        state["world"] = pkg.VecGridWorld(pkg.make_config(case["width"], case["height"], case["envs"], 0xC0DA2025 + seed, obstacle_kind=pkg.OBST_BERNOULLI,
                                                          obstacle_p=case["p"], goal_mode=pkg.GOAL_SEEDED, num_goals=1, start_mode=pkg.START_RANDOM))
        state["actions"] = rng.integers(0, 4, case["envs"]).astype(np.int32)
        state["world"].step_actions(state["actions"])
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "env":
        env = state["env"]
        env.reset()
        rewards, dones, places = [], [], []
        for action in state["actions"]:
            observation, reward, done, _info = env.step(action)
            rewards.append(reward)
            dones.append(done)
            places.append(env.get_agent_position())
            if done:
                env.reset()
        return np.asarray(rewards, np.float32), np.asarray(dones, np.uint8), np.asarray(places, np.int32), np.asarray(observation, np.float32)
    world = state["world"]
    if case["kind"] == "train":
        if "eps" in state:
            world.train_steps_eps(state["eps"])
        else:
            world.train_steps(case["steps"])
        q, (x, y, t), s = world.get_q(), world.get_state(), world.get_stats()
        return dict(q=q, x=x, y=y, t=t, steps=s.steps, episodes=s.episodes, goals=s.goals, timeouts=s.timeouts, conflicts=s.conflicts,
                    long_chains=s.long_chains, chained=s.chained, reward_sum=s.reward_sum, epsilon=s.epsilon)
    if case["kind"] == "eval":
        s = world.eval_rollout(case["steps"])
        return dict(envs=s.envs, reached=s.reached, total_steps=s.total_steps, reward_sum=s.reward_sum)
    if case["kind"] == "update":
        for batch in state["batches"]:
            world.update_batch(*batch)
        return world.get_q()
    rewards, dones = world.step_actions(state["actions"])
    x, y, t = world.get_state()
    return rewards, dones, x, y, t


def work(case):
    cells = case["width"] * case["height"]
    if case["kind"] == "env":                        # per step: the action in, position, reward, done flag and the observed grid out
        return dict(bytes=case["steps"] * (4 + 13 + 4 * cells), flops=case["steps"])
    if case["kind"] == "train":
        # one batched step: every state in and out (12 bytes each way), the rows of the current and the next cell in and the updated
        # entry out -- but no table row more than once; the steps follow one another; table and states out at the end
        n = case["envs"]
        step = 24 * n + min(32 * n, 16 * cells) + min(4 * n, 16 * cells)
        return dict(bytes=case["steps"] * step + 16 * cells + 12 * n, flops=case["steps"] * 4 * n)
    if case["kind"] == "eval":                       # the table and the cell classes in once; a start cell for every environment
        return dict(bytes=17 * cells + 4 * case["envs"], flops=3 * cells)
    if case["kind"] == "update":                     # the transitions in, the rows they touch in, the entries out; the table out
        n = case["batch"]
        return dict(bytes=case["calls"] * (25 * n + min(32 * n, 16 * cells) + min(4 * n, 16 * cells)) + 16 * cells, flops=case["calls"] * 4 * n)
    return dict(bytes=case["envs"] * (4 + 12 + 12 + 2 + 5 + 12), flops=case["envs"])   # action, state in and out, cell class, reward and flag, state read


def tolerance(case):
    return "exact"
