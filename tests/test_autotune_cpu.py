"""What the autotuner tries and what it remembers, with a stand-in for the env
and the clock (no GPU)."""
import contextlib

import pytest

from minecu import autotune, capi

KEYS = ("stage", "warps_per_cta", "ctas_per_sm", "tile_w", "team_warps", "coop")


class FakeEnv:
    """An env whose step time is a function of its launch shape."""
    device = "cpu"
    batch_size, obs_dtype, numerics = 64, "uint8", "ref_fast"
    world_x = world_y = world_z = 16
    render_width = render_height = 32
    max_steps, view_distance = 64, 32.0

    def __init__(self, shape, cost):
        self.shape, self.cost, self.timed = tuple(shape), cost, []

    def launch_config(self):
        return dict(zip(KEYS, self.shape), smem_bytes=0)

    def set_launch_config(self, *c):
        self.shape = tuple(c)

    def rollout(self, *a):
        self.timed.append(self.shape)

    def state_dict(self):
        return {}

    def reset(self):
        pass

    prepare_rollout = load_state_dict = check_error = lambda self, *a: None


@pytest.fixture
def clock(monkeypatch, tmp_path):
    monkeypatch.setenv("MINECU_TUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(autotune.torch.cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(autotune, "_device_key", lambda d: "dev")
    monkeypatch.setattr(autotune, "_actions", lambda n, steps, seed, d: list(range(steps)))
    now = {}

    def window(run, restore, reps=2):
        run()
        return now["env"].cost(now["env"].shape)

    monkeypatch.setattr(autotune, "_time_window", window)
    return now


def _default_shape(B, image=32, world=16):
    import ctypes
    c = capi.make_config(B, world, world, world, image, image)
    f = capi.FusedConfig()
    capi.check(capi.lib().mc_default_fused_config(ctypes.byref(c), 148, 1, ctypes.byref(f), None), "default")
    return tuple(getattr(f, k) for k in KEYS)


@pytest.mark.parametrize("B", [1, 16, 64, 256, 1024, 32768])
def test_tuning_never_ends_slower_than_the_shape_it_found(clock, B):
    start = _default_shape(B)
    clock["env"] = env = FakeEnv(start, lambda s: 1.0 if s == start else 2.0)
    out = autotune.tune_env(env, steps=2, warm_steps=1)
    assert tuple(out["config"]) == start == env.shape and out["ms_per_step"] == 0.5


@pytest.mark.parametrize("B", [1, 16, 64, 256, 1024, 4096])
def test_the_tuner_tries_every_tile_width_the_defaults_use(B):
    tiles = {c[3] for c in autotune.env_candidates()}
    assert _default_shape(B)[3] in tiles


def test_no_two_candidates_are_the_same_launch():
    """With one warp per env a staging depth of 2 is one of 1."""
    launches = [c if c[5] or c[4] > 1 else (min(c[0], 1),) + tuple(c[1:]) for c in autotune.env_candidates()]
    assert len(set(launches)) == len(launches)


def test_shapes_tuned_for_other_kernels_are_measured_again(clock, monkeypatch, tmp_path):
    slow, quick = (0, 8, 4, 4, 1, 0), (1, 8, 3, 8, 4, 1)
    libs = []
    for k in range(2):
        libs.append(tmp_path / f"lib{k}.so")
        libs[k].write_bytes(b"kernels %d" % k)
    cands = [slow, quick]
    monkeypatch.setattr(capi, "LIB_PATH", str(libs[0]))
    clock["env"] = env = FakeEnv(slow, lambda s: 1.0 if s == slow else 2.0)
    assert tuple(autotune.tune_env(env, steps=2, warm_steps=1, candidates=cands)["config"]) == slow
    clock["env"] = env = FakeEnv(slow, lambda s: 1.0 if s == quick else 2.0)
    assert tuple(autotune.tune_env(env, steps=2, warm_steps=1, candidates=cands)["config"]) == slow  # remembered
    monkeypatch.setattr(capi, "LIB_PATH", str(libs[1]))  # other kernels
    assert tuple(autotune.tune_env(env, steps=2, warm_steps=1, candidates=cands)["config"]) == quick
    batch = type("Batch", (), dict(device="cpu", envs=[env]))()
    other = autotune._ragged_key(batch)
    monkeypatch.setattr(capi, "LIB_PATH", str(libs[0]))
    assert autotune._ragged_key(batch) != other
