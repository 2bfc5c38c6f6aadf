"""The fused form's agent and image kernels at the edges of their dispatch,
against the CPU oracle (ieee numerics, no tolerance): batches around the agent
kernel's block size, images cut into slices, more units than the grid has
warps (records filed marching envs first), worlds regenerated by the image
warps under both rules, and the images of resets, which come from the same
kernels."""
import numpy as np
import pytest

from minecu import capi
import oracle as O
from mc_harness import GpuEnv, actions_for, diff_report, oracle_state

pytestmark = pytest.mark.gpu


def run(cuda, B, steps, seed, world=(16, 16, 16), res=(32, 32), regen="all", cfg=None, reset_every=3, break_half=True,
        **kw):
    g = GpuEnv(cuda, B, world_x=world[0], world_y=world[1], world_z=world[2], render_width=res[0],
               render_height=res[1], debug=False, **kw)
    if cfg:
        g.set_fused(*cfg)
    if regen != "all":
        g.set_regen(True)
    o = O.OracleEnv(batch_size=B, world_x=world[0], world_y=world[1], world_z=world[2], render_width=res[0],
                    render_height=res[1], regen=regen, **kw)
    g.reset()
    o.reset()
    rng = np.random.default_rng(seed)

    def same(what):
        d = diff_report(g.state(), oracle_state(o))
        assert not d, f"{what}: {d}"

    same("reset")
    for s in range(steps):
        _, btn, look = actions_for(B, s, seed, 0.1, break_half)
        btn[:, 6] = rng.random(B) < 0.1
        g.step(btn, look, capi.FORM_FUSED)
        o.step(btn, look)
        same(f"step {s}")
        if reset_every and s % reset_every == reset_every - 1:
            mask = rng.random(B) < (0.3 if B > 1 else 1.0)
            g.reset(mask)
            o.reset(mask)
            same(f"masked reset after step {s}")
    g.check_error()
    g.close()


@pytest.mark.parametrize("regen", ["all", "per_env"])
@pytest.mark.parametrize("B", [1, 2, 127, 128, 129, 300])
def test_batch_edges(cuda, B, regen):
    run(cuda, B, 12, 40 + B, regen=regen, obs_dtype="uint8", episode_length=5)


@pytest.mark.parametrize("mode", ["float32", "uint8_minimal", "uint8_prebasis_full", "uint8_fp16", "uint8_fast"])
def test_reset_images_of_every_mode(cuda, mode):
    run(cuda, 33, 9, 51, obs_dtype=mode, episode_length=4)
    run(cuda, 5, 4, 52, world=(32, 32, 32), res=(64, 64), obs_dtype=mode, episode_length=3, regen="per_env")


@pytest.mark.parametrize("regen", ["all", "per_env"])
def test_records_filed_by_cost(cuda, regen):
    """More units than warps: marching envs from the front, buried ones from the back."""
    run(cuda, 10007, 16, 53, res=(8, 8), regen=regen, obs_dtype="uint8", episode_length=13, reset_every=7)


@pytest.mark.parametrize("cfg", [(1, 8, 3, 8, 4, 1), (2, 8, 2, 8, 4, 1), (1, 8, 3, 16, 8, 1), (1, 8, 3, 8, 2, 0)],
                         ids=["team", "team_depth2", "team8", "per_warp_groups"])
@pytest.mark.parametrize("regen", ["all", "per_env"])
def test_team_images(cuda, cfg, regen):
    run(cuda, 3, 8, 54, res=(64, 64), regen=regen, cfg=cfg, obs_dtype="uint8", episode_length=4)
    run(cuda, 41, 8, 55, world=(32, 16, 32), res=(32, 32), regen=regen, cfg=cfg, obs_dtype="uint8", episode_length=4)


@pytest.mark.parametrize("res", [(1, 1), (7, 5), (31, 33), (84, 84), (17, 64), (40, 9)])
@pytest.mark.parametrize("cfg", [(1, 8, 4, 4, 1, 0), (1, 8, 3, 8, 4, 1), (1, 8, 2, 32, 2, 0)],
                         ids=["per_warp", "team", "per_warp_groups"])
def test_odd_images(cuda, res, cfg):
    """Images that are no whole tiles, whose rows and envs start at any byte."""
    for mode in ("uint8", "float32", "uint8_prebasis"):
        run(cuda, 5, 6, 56, res=res, cfg=cfg, obs_dtype=mode, episode_length=4)


@pytest.mark.parametrize("world", [(5, 5, 5), (9, 40, 13), (7, 11, 23), (26, 33, 21), (16, 16, 17), (33, 9, 40)])
@pytest.mark.parametrize("cfg", [None, (0, 8, 4, 8, 1, 0), (0, 8, 3, 8, 4, 1), (0, 8, 2, 8, 2, 0)],
                         ids=["default", "per_warp", "team", "per_warp_groups"])
def test_worlds_of_any_size(cuda, world, cfg):
    """Worlds of no whole 16-byte chunks (every env's starts at another byte), staged by their chunks and edges."""
    for mode in ("uint8", "uint8_minimal"):
        run(cuda, 9, 7, 57, world=world, res=(24, 16), cfg=cfg, obs_dtype=mode, episode_length=4,
            ground_height=min(8, world[1] // 2), regen="per_env")


def test_voxels_at_any_byte(cuda):
    """A voxels view that starts off a 16-byte boundary."""
    import ctypes
    import torch
    B = 6
    g = GpuEnv(cuda, B, debug=False, obs_dtype="uint8", episode_length=4)
    base = torch.empty(B * 4096 + 32, dtype=torch.int8, device=cuda)
    view = base[3:3 + B * 4096].view(B, 16, 16, 16)
    g.t["voxels"] = view
    g.st.voxels = view.data_ptr()
    capi.check(g.L.mc_env_set_state(g.h, ctypes.byref(g.st)), "set_state")
    g.set_fused(0, 8, 4, 4, 1, 0)
    capi.check(g.L.mc_env_generate_world(g.h, None), "generate_world")
    o = O.OracleEnv(batch_size=B, obs_dtype="uint8", episode_length=4, world_size=16, render_width=32, render_height=32)
    g.reset()
    o.reset()
    for s in range(9):
        _, btn, look = actions_for(B, s, 58, 0.1, True)
        g.step(btn, look, capi.FORM_FUSED)
        o.step(btn, look)
        d = diff_report(g.state(), oracle_state(o))
        assert not d, f"step {s}: {d}"
    g.check_error()
    g.close()


@pytest.mark.parametrize("world", [(40, 40, 40), (41, 39, 43), (48, 48, 48), (56, 56, 56), (64, 56, 64)])
def test_big_worlds(cuda, world):
    """Worlds above 32 KB, with the default launch shape (as many staged worlds as an SM holds, or none)."""
    run(cuda, 5, 5, 59, world=world, res=(64, 48), obs_dtype="uint8", episode_length=3, regen="per_env")
    run(cuda, 2, 4, 60, world=world, res=(31, 20), obs_dtype="uint8_minimal", episode_length=3)


@pytest.mark.parametrize("mode", ["uint8_fast", "uint8_fp16"])
@pytest.mark.parametrize("kw", [dict(), dict(world=(32, 32, 32), res=(64, 64)), dict(world=(9, 20, 13), res=(21, 17)),
                                dict(max_steps=20, view_distance=6.0), dict(max_steps=3, view_distance=2.5),
                                dict(world=(24, 16, 20), ground_height=4, max_steps=61),
                                dict(world=(6, 24, 6), res=(48, 48), ground_height=2, max_steps=37),
                                dict(world=(16, 16, 16), ground_height=0)],
                         ids=lambda k: "_".join(f"{a}{b}" for a, b in k.items()).replace(" ", "") or "c1")
def test_ground_shortcut_and_fp16(cuda, mode, kw):
    """The fast marches of the ground-shortcut and binary16 families: rays that
    enter the ground, leave the box sideways above it, run out of steps or of
    view."""
    for cfg in (None, (1, 8, 3, 8, 4, 1)):
        if cfg and (np.prod(kw.get("world", (16, 16, 16))) % 16):
            cfg = (0,) + cfg[1:]
        run(cuda, 14, 10, 61, obs_dtype=mode, cfg=cfg, episode_length=7, regen="per_env", **kw)


@pytest.mark.parametrize("mode", ["uint8", "uint8_prebasis"])
def test_images_too_wide_for_a_fused_launch(cuda, mode):
    """Rows whose bands fit no launch shape's shared memory: resets and renders still work, beside plain steps."""
    B = 2
    kw = dict(world_x=16, world_y=16, world_z=16, render_width=20000, render_height=2, obs_dtype=mode, episode_length=2)
    g = GpuEnv(cuda, B, debug=False, **kw)
    o = O.OracleEnv(batch_size=B, **kw)
    g.reset()
    o.reset()
    assert not diff_report(g.state(), oracle_state(o))
    for s in range(4):
        _, btn, look = actions_for(B, s, 62, 0.1, True)
        g.step(btn, look, capi.FORM_PLAIN)
        o.step(btn, look)
        assert not diff_report(g.state(), oracle_state(o)), s
        mask = np.array([s % 2 == 0, False])
        g.reset(mask)
        o.reset(mask)
        assert not diff_report(g.state(), oracle_state(o)), s
    g.close()


@pytest.mark.parametrize("B", [1, 45])
@pytest.mark.parametrize("n", [1, 4, 5, 12, 13, 32])
def test_interactions_per_warp(cuda, B, n):
    """n envs of each warp break or place: up to 12 share the warp's lanes, more take a thread each."""
    kw = dict(world_x=16, world_y=16, world_z=16, render_width=32, render_height=32, obs_dtype="uint8", episode_length=9)
    g = GpuEnv(cuda, B, debug=False, **kw)
    o = O.OracleEnv(batch_size=B, **kw)
    g.reset()
    o.reset()
    rng = np.random.default_rng(63)
    for s in range(14):
        _, btn, look = actions_for(B, s, 63, 0.1, False)
        look = (look + rng.normal(0, 0.3, look.shape)).astype(np.float32)
        act = (np.arange(B) + 3 * s) % 32 < n
        btn[:, 5] = act & (rng.random(B) < 0.7)
        btn[:, 6] = act & (btn[:, 5] == 0)
        g.step(btn, look, capi.FORM_FUSED)
        o.step(btn, look)
        d = diff_report(g.state(), oracle_state(o))
        assert not d, f"step {s}: {d}"
    g.check_error()
    g.close()
