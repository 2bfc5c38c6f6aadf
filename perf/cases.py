"""The work that programs have this framework do, as cases that can be timed.

A case is a dict of plain values.  `kind` says which public entry points one
pass goes through:

  step     MineEnv.step, discrete actions or buttons + look, device tensors
  host     MineEnv.step_host + join_host, a policy on the host
  rollout  MineEnv.reset, then MineEnv.rollout: whole episodes in one graph
  reset    MineEnv.step, reset(mask) of the envs the trainer ends itself, and
           policy_obs, the float32 input of its network
  ragged   RaggedBatch.step over groups of different worlds and images
  serve    one request of every client job of an EnvServer

Steps run where a trainer's steps run: in the middle of episodes.  `prepare`
spreads the envs over their episode (independent episodes, regen="per_env")
and steps them through one, so every pass sees the same mix of agents that
fall, stand, dig and look around, whatever the number of passes before it.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mine.cu_b200"))

from minecu import MineEnv  # noqa: E402
from minecu.ragged import RaggedBatch  # noqa: E402
from minecu.server import EnvServer  # noqa: E402

MODES = ("uint8", "float32", "uint8_minimal", "uint8_prebasis", "uint8_prebasis_full", "uint8_smem", "uint8_fp16",
         "uint8_fast")
POOL = 61  # action sets that a state keeps and takes in turn
BREAK = 6  # the discrete action "break"


def _case(name, kind, batch, world, image, mode="uint8", *, act="discrete", break_half=False, episode=60, ground=8,
          max_steps=64, view=32.0, steps=1, regen="per_env"):
    wx, wy, wz = world if isinstance(world, tuple) else (world,) * 3
    w, h = image if isinstance(image, tuple) else (image,) * 2
    c = dict(kind=kind, batch=batch, world_x=wx, world_y=wy, world_z=wz, width=w, height=h, mode=mode, act=act,
             break_half=break_half, episode=episode, ground=ground, max_steps=max_steps, view=view, steps=steps,
             regen=regen)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # one env: an evaluation, a recording, a debugging session
        _case("single_env", "step", 1, 16, 64),
        # the small batch of the reference's plain method, 64 envs
        _case("small_batch", "step", 64, 16, 32),
        # a PPO-sized batch with the reference's own action form
        _case("trainer_1k", "step", 1024, 16, 64, act="buttons", episode=240),
        # the peak shape (32768 envs, 16^3, 32x32), long episodes
        _case("peak", "step", 32768, 16, 32, episode=240),
        # the same shape with MineEnv's default observation type
        _case("peak_float32", "step", 32768, 16, 32, "float32"),
        # render-dominated: 32^3 worlds, 64x64, half of the actions break blocks
        _case("render", "step", 4096, 32, 64, break_half=True),
        # odd sizes: a world of three different edges, 84x84 images as Atari-style networks take them, and the
        # observation mode whose episodes the kernel keeps
        _case("odd_sizes", "step", 1500, (24, 16, 20), 84, "uint8_prebasis_full", act="buttons"),
        # the QUALITY preset: 128x128 float32 images, 128 steps a ray
        _case("quality_preset", "step", 4096, 32, 128, "float32", max_steps=128, view=64.0),
        # the FAST preset's episode, 60 steps from a reset, the reference's rule for worlds (32^3 by default)
        _case("fast_preset_episode", "rollout", 32768, 32, 32, max_steps=32, steps=60, regen="all"),
        # a host-side policy: pinned actions in, rewards and dones out
        _case("host_policy", "host", 4096, 16, 32, episode=240),
        # a trainer that ends episodes itself and feeds a network
        _case("masked_reset", "reset", 4096, 16, 64),
        # 24,576 envs in six groups of different worlds and images, one launch
        dict(name="ragged_six", kind="ragged", groups="8192:8:16 6144:16:32 4096:16:64 3072:24:32 2048:32:32 1024:32:64",
             mode="uint8", act="discrete", break_half=False, episode=60),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _world(rng):
    if rng.random() < 0.6:
        e = rng.choice((8, 12, 16, 16, 16, 20, 24, 32, 32, 40, 48))
        return (e, e, e)
    return (_log_int(rng, 6, 48), _log_int(rng, 6, 40), _log_int(rng, 6, 48))


def _image(rng):
    if rng.random() < 0.5:
        e = rng.choice((16, 24, 32, 32, 48, 64, 64, 84, 96, 128))
        return (e, e)
    return (_log_int(rng, 7, 128), _log_int(rng, 7, 128))


def draw(rng):
    kind = rng.choice(("step",) * 12 + ("host", "host", "rollout", "rollout", "reset", "reset", "ragged", "ragged", "serve"))
    mode = rng.choice(("uint8",) * 6 + ("float32",) * 4 + MODES[2:])
    if kind in ("ragged", "serve"):
        groups = []
        for _ in range(rng.randint(2, 8)):
            e, r = rng.choice((8, 12, 16, 16, 24, 32)), rng.choice((16, 24, 32, 32, 48, 64))
            groups.append("%d:%d:%d" % (_log_int(rng, 32, 4096), e, r))
        return dict(kind=kind, groups=" ".join(groups), mode="uint8" if kind == "serve" else mode,
                    act="discrete" if kind == "serve" else rng.choice(("discrete", "buttons")),
                    break_half=rng.random() < 0.3, episode=rng.choice((60, 120)))
    world, image = _world(rng), _image(rng)
    most = min(32768, int(4.0e7 / (image[0] * image[1])), int(5.0e8 / (world[0] * world[1] * world[2])))
    steps = 1
    if kind == "rollout":
        steps = _log_int(rng, 4, 60)
        most = max(1, min(most, int(3.0e8 / (steps * image[0] * image[1]))))
    batch = _log_int(rng, 1, most)
    return _case(None, kind, batch, world, image, mode,
                 act="discrete" if kind in ("host", "rollout") else rng.choice(("discrete", "discrete", "buttons")),
                 break_half=rng.random() < 0.3, episode=rng.choice((30, 60, 60, 120)),
                 ground=min(8, max(2, world[1] // 2)), max_steps=rng.choice((32, 64, 64, 128)),
                 view=rng.choice((16.0, 32.0, 32.0, 64.0)), steps=steps, regen="all" if kind == "rollout" else "per_env")


def _groups(case):
    """(batch, world edge, image edge, ground height) of each group or job."""
    return [(b, e, r, min(8, max(2, e // 2))) for b, e, r in (map(int, g.split(":")) for g in case["groups"].split())]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _actions(case, total, count, g):
    """`count` action sets for `total` envs: uint8 [count, total], or (buttons, look)."""
    if case["act"] == "discrete":
        a = torch.randint(0, 11, (count, total), generator=g, device="cuda", dtype=torch.uint8)
        if case["break_half"]:
            a[torch.rand((count, total), generator=g, device="cuda") < 0.5] = BREAK
        return a
    # a policy's multi-hot buttons: forward and break often, the others less
    p = torch.tensor([0.5, 0.1, 0.15, 0.15, 0.1, 0.5 if case["break_half"] else 0.2, 0.05, 0.2], device="cuda")
    b = (torch.rand((count, total, 8), generator=g, device="cuda") < p).to(torch.int8)
    look = torch.randn((count, total, 2), generator=g, device="cuda") * 0.1
    return [(b[k], look[k]) for k in range(count)]


def _spread(batch, episode, seed):
    """Where in its episode each env is at first (its step count)."""
    return (torch.randint(0, episode, (batch,), generator=_generator(seed + 1000003), device="cuda")).to(torch.int32)


def _make_env(case, seed):
    env = MineEnv(batch_size=case["batch"], world_x=case["world_x"], world_y=case["world_y"], world_z=case["world_z"],
                  render_width=case["width"], render_height=case["height"], max_steps=case["max_steps"],
                  view_distance=case["view"], ground_height=case["ground"], episode_length=case["episode"],
                  obs_dtype=case["mode"], regen=case["regen"])
    env.reset()
    return env


def _take(state):
    k = state["next"]
    state["next"] = (k + 1) % len(state["actions"])
    return state["actions"][k]


def _step(target, a):
    return target.step(*a) if isinstance(a, tuple) else target.step(a)


def _env_state(env):
    return {k: getattr(env, k) for k in ("voxels", "positions", "velocities", "yaws", "pitches", "on_ground", "step_count",
                                         "cameras")}


def prepare(case, seed):
    g = _generator(seed)
    kind, episode = case["kind"], case["episode"]
    if kind == "ragged":
        groups = _groups(case)
        envs = [MineEnv(batch_size=b, world_size=e, render_width=r, render_height=r, ground_height=gh,
                        episode_length=episode, obs_dtype=case["mode"], regen="per_env") for b, e, r, gh in groups]
        batch = RaggedBatch(envs)
        batch.reset()
        for i, env in enumerate(envs):
            env.step_count.copy_(_spread(env.batch_size, episode, seed + i))
        state = dict(kind=kind, batch=batch, next=0, actions=_actions(case, batch.total, POOL, g))
        for _ in range(episode):
            _step(batch, _take(state))
        return state
    if kind == "serve":
        server = EnvServer(hbm_budget_bytes=20e9)
        jobs = [server.admit(b, world_size=e, render_width=r, render_height=r, ground_height=gh, episode_length=episode)
                for b, e, r, gh in _groups(case)]
        pool = [list(_actions(case, b, POOL, g).cpu()) for b, _, _, _ in _groups(case)]
        for job in jobs:
            server.reset(job)
        state = dict(kind=kind, server=server, jobs=jobs, next=0, actions=list(zip(*pool)),
                     views=[server.state(j) for j in jobs])
        for _ in range(24):
            _serve(state)
        return state
    env = _make_env(case, seed)
    state = dict(kind=kind, env=env, next=0)
    if kind == "rollout":
        state["actions"] = _actions(case, case["batch"], case["steps"], g)
        state["rewards"] = torch.empty((case["steps"], case["batch"]), dtype=torch.float32, device="cuda")
        state["dones"] = torch.empty((case["steps"], case["batch"]), dtype=torch.bool, device="cuda")
        env.prepare_rollout(state["actions"], state["rewards"], state["dones"])
        return state
    state["actions"] = _actions(case, case["batch"], POOL, g)
    env.step_count.copy_(_spread(case["batch"], episode, seed))
    for _ in range(episode):
        _step(env, _take(state))
    if kind == "host":
        host = torch.empty((POOL, case["batch"]), dtype=torch.uint8, pin_memory=True)
        host.copy_(state["actions"])
        state["actions"] = host
        state["rewards"] = torch.empty(case["batch"], dtype=torch.float32, pin_memory=True)
        state["dones"] = torch.empty(case["batch"], dtype=torch.bool, pin_memory=True)
    if kind == "reset":
        state["masks"] = torch.rand((POOL, case["batch"]), generator=g, device="cuda") < 0.03
        shape = (case["batch"], 3, case["height"], case["width"])
        state["policy"] = torch.empty(shape, dtype=torch.float32, device="cuda")
    return state


def _serve(state):
    row = _take(state)
    tickets = [state["server"].submit(j, a) for j, a in zip(state["jobs"], row)]
    return [state["server"].wait(t) for t in tickets]


def run(state):
    kind = state["kind"]
    if kind == "step":
        env = state["env"]
        obs, rewards, dones = _step(env, _take(state))
        return dict(obs=obs, rewards=rewards, dones=dones, state=_env_state(env))
    if kind == "host":
        env = state["env"]
        obs = env.step_host(_take(state), state["rewards"], state["dones"])
        env.join_host()
        return dict(obs=obs, rewards=state["rewards"], dones=state["dones"], state=_env_state(env))
    if kind == "rollout":
        env = state["env"]
        env.reset()
        env.rollout(state["actions"], state["rewards"], state["dones"])
        return dict(obs=env.obs_buffer, rewards=state["rewards"], dones=state["dones"], state=_env_state(env))
    if kind == "reset":
        env = state["env"]
        mask = state["masks"][state["next"]]
        _, rewards, dones = _step(env, _take(state))
        obs = env.reset(mask)
        return dict(obs=obs, rewards=rewards, dones=dones, policy=env.policy_obs(out=state["policy"]),
                    state=_env_state(env))
    if kind == "ragged":
        return [dict(obs=o, rewards=r, dones=d, positions=e.positions, voxels=e.voxels)
                for (o, r, d), e in zip(_step(state["batch"], _take(state)), state["batch"].envs)]
    results = _serve(state)
    return [dict(obs=v["obs"], rewards=r, dones=d, positions=v["positions"], voxels=v["voxels"])
            for (r, d), v in zip(results, state["views"])]


def _one_step(case, batch, world, image):
    """Bytes and operations of one step of a batch: each world and each agent read once, each image, agent and result
    written once; per ray its direction, the entry to the first voxel, a few voxels and the colour."""
    pixels = image[0] * image[1]
    channel = 4 if case["mode"] == "float32" else 1
    action = 1 if case["act"] == "discrete" else 16
    agent = 12 + 12 + 4 + 4 + 1 + 4
    moved = batch * (world[0] * world[1] * world[2] + pixels * 3 * channel + 2 * agent + 20 + 4 + 1 + action)
    return moved, batch * pixels * 70.0


def work(case):
    if case["kind"] in ("ragged", "serve"):
        parts = [_one_step(case, b, (e, e, e), (r, r)) for b, e, r, _ in _groups(case)]
        return dict(bytes=sum(p[0] for p in parts), flops=sum(p[1] for p in parts))
    world = (case["world_x"], case["world_y"], case["world_z"])
    image = (case["width"], case["height"])
    moved, flops = _one_step(case, case["batch"], world, image)
    voxels, pixels = world[0] * world[1] * world[2], image[0] * image[1]
    channel = 4 if case["mode"] == "float32" else 1
    if case["kind"] == "rollout":  # the worlds and images of the reset, then the steps
        return dict(bytes=case["steps"] * moved + case["batch"] * (voxels + pixels * 3 * channel),
                    flops=(case["steps"] + 1) * flops)
    if case["kind"] == "reset":  # the step, the images after the reset, and the policy's input
        return dict(bytes=moved + case["batch"] * pixels * 3 * (2 * channel + 4), flops=2 * flops)
    return dict(bytes=moved, flops=flops)


def exact(case, seed):
    """The agents of a single batch in 64 bits (they move over flat ground, whatever the worlds hold).  What depends on
    worlds (images, rewards, voxels) has no value in other arithmetic: a ray that grazes an edge meets another block."""
    if case["kind"] not in ("step", "host"):
        return None
    n, episode, f8 = case["batch"], case["episode"], torch.float64
    actions = _actions(case, n, POOL, _generator(seed))
    count = _spread(n, episode, seed).to(torch.int64)
    spawn = torch.tensor([case["world_x"] / 2, case["ground"] + 2.0, case["world_z"] / 2], dtype=f8, device="cuda")
    high = torch.tensor([case["world_x"] - 1.0, 0.0, case["world_z"] - 1.0], dtype=f8, device="cuda")
    f32 = lambda v: float(torch.tensor(v, dtype=torch.float32))  # noqa: E731
    dt, pitch_most, turn, floor = f32(0.05), f32(1.56), f32(0.1), float(case["world_y"] // 4)
    pos, vy = spawn.repeat(n, 1), torch.zeros(n, dtype=f8, device="cuda")
    yaw, pitch = torch.zeros(n, dtype=f8, device="cuda"), torch.zeros(n, dtype=f8, device="cuda")
    ground = torch.zeros(n, dtype=torch.bool, device="cuda")
    for t in range(episode + 1):
        a = actions[t % POOL]
        if isinstance(a, tuple):
            b, look = a[0].to(f8), a[1].to(f8)
            forward, strafe, jump = b[:, 0] - b[:, 1], b[:, 3] - b[:, 2], b[:, 4] != 0
            speed = torch.where((b[:, 0] != 0) & (b[:, 7] != 0), 1.5, 1.0).to(f8)
            dyaw, dpitch = look[:, 0], look[:, 1]
        else:
            forward = (a == 1).to(f8) - (a == 2).to(f8)
            strafe = (a == 4).to(f8) - (a == 3).to(f8)
            jump, speed = a == 5, torch.ones(n, dtype=f8, device="cuda")
            dyaw = turn * ((a == 7).to(f8) - (a == 8).to(f8))
            dpitch = turn * ((a == 9).to(f8) - (a == 10).to(f8))
        yaw = yaw + dyaw
        pitch = (pitch + dpitch).clamp(-pitch_most, pitch_most)
        sin, cos = torch.sin(yaw), torch.cos(yaw)
        dx = (sin * forward * speed + cos * strafe) * 4.0 * dt
        dz = (cos * forward * speed - sin * strafe) * 4.0 * dt
        vy = torch.where(jump & ground, 8.0, vy) - 20.0 * dt
        y = pos[:, 1] + vy * dt
        ground = y <= floor
        y, vy = torch.where(ground, floor, y), torch.where(ground, 0.0, vy)
        x = torch.minimum((pos[:, 0] + dx).clamp(min=1.0), high[0])
        z = torch.minimum((pos[:, 2] + dz).clamp(min=1.0), high[2])
        pos = torch.stack([x, y, z], 1)
        done = count >= episode
        count = torch.where(done, 1, count + 1)
        pos = torch.where(done[:, None], spawn, pos)
        vy, yaw, pitch = (torch.where(done, 0.0, v) for v in (vy, yaw, pitch))
        ground = ground & ~done
    still = torch.zeros_like(vy)
    state = dict(voxels=None, positions=pos, velocities=torch.stack([still, vy, still], 1), yaws=yaw, pitches=pitch,
                 on_ground=None, step_count=None, cameras=torch.cat([pos, yaw[:, None], pitch[:, None]], 1))
    return dict(obs=None, rewards=None, dones=None, state=state)
