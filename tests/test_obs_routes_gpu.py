"""Images of reset() and get_obs() by both of their routes (the step's image
kernels, and a thread a pixel): envs on either side of each line between them,
and a handle whose launch shape and buffers change, against the CPU oracle."""
import ctypes

import numpy as np
import pytest

from minecu import capi
import oracle as O
from mc_harness import GpuEnv, actions_for, diff_report, oracle_state

pytestmark = pytest.mark.gpu


def _pair(cuda, B, world, res, **kw):
    kw = dict(world_x=world[0], world_y=world[1], world_z=world[2], render_width=res[0], render_height=res[1],
              ground_height=min(8, world[1] // 2), **kw)
    g = GpuEnv(cuda, B, debug=False, numerics="ieee", **kw)
    return g, O.OracleEnv(batch_size=B, **kw)


def _same(g, o, what):
    d = diff_report(g.state(), oracle_state(o))
    assert not d, f"{what}: {d}"


def _walk(g, o, B, seed, steps=3):
    rng = np.random.default_rng(seed)
    g.reset()
    o.reset()
    _same(g, o, "reset")
    for s in range(steps):
        _, btn, look = actions_for(B, s, seed, 0.1, True)
        g.step(btn, look, capi.FORM_FUSED)
        o.step(btn, look)
        mask = rng.random(B) < 0.5
        g.reset(mask)
        o.reset(mask)
        _same(g, o, f"masked reset {s}")
        g.t["obs"].zero_()
        g.render()  # the images a reset left are those of the state
        _same(g, o, f"get_obs {s}")


@pytest.mark.parametrize("mode", ["uint8", "float32"])
@pytest.mark.parametrize("B, world, res", [(1, (16, 16, 16), (32, 32)), (1, (16, 16, 16), (84, 84)),
                                           (1, (9, 40, 13), (120, 64)), (64, (16, 16, 16), (64, 64)),
                                           (40, (16, 16, 16), (84, 84)), (3, (48, 48, 48), (8, 8)),
                                           (2, (70, 16, 66), (24, 20)), (2, (64, 64, 64), (32, 32)),
                                           (1100, (16, 16, 16), (8, 8)),
                                           (180, (66, 24, 60), (160, 152))])
def test_images_of_both_routes(cuda, mode, B, world, res):
    g, o = _pair(cuda, B, world, res, obs_dtype=mode)
    _walk(g, o, B, 121)
    g.close()


def test_the_route_follows_the_shape_and_the_state(cuda):
    """Both routes on one handle: staged, unstaged (no common path), and with an image buffer off its alignment."""
    import torch
    B, res = 5, (32, 32)
    g, o = _pair(cuda, B, (16, 16, 16), res, obs_dtype="uint8")
    _walk(g, o, B, 122, 2)
    g.set_fused(0, 8, 4, 8, 1, 0)
    _walk(g, o, B, 123, 2)
    g.set_fused(1, 8, 3, 8, 4, 1)
    _walk(g, o, B, 124, 2)
    n = B * res[0] * res[1] * 3
    base = torch.zeros(n + 16, dtype=torch.uint8, device=cuda)
    g.t["obs"] = base[5:5 + n].view(B, res[1], res[0], 3)
    g.st.obs = g.t["obs"].data_ptr()
    capi.check(g.L.mc_env_set_state(g.h, ctypes.byref(g.st)), "set_state")
    _walk(g, o, B, 125, 2)
    g.close()
