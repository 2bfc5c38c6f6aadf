"""Small worlds just beyond the packed march's index field, with solid voxels in
their top layer (the tree's leaves or the house's roof reach it), seen by eyes
that look up: their rays leave through the top, whose voxels the march loads
before it sees that it has left.  These worlds take the split march.  Against
the CPU oracle, bit for bit, in the normal and the bounds-checked build."""
import ctypes

import numpy as np
import pytest

from minecu import capi
import oracle as O
from mc_harness import GpuEnv, diff_report, oracle_state

pytestmark = pytest.mark.gpu

WORLDS = {(31, 8, 31): 4, (25, 13, 25): 8, (27, 11, 27): 6, (20, 20, 20): 15, (28, 10, 28): 6}  # ground height
MODES = ["uint8", "float32", "uint8_minimal", "uint8_prebasis", "uint8_fp16", "uint8_fast"]


@pytest.mark.parametrize("checked", [True, False], ids=["checked", "normal"])
@pytest.mark.parametrize("world", sorted(WORLDS), ids=lambda w: "x".join(map(str, w)))
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("cfg", [(1, 8, 4, 4, 1, 0), (1, 8, 3, 8, 4, 1)], ids=["per_warp", "team"])
def test_rays_leave_through_a_solid_top_layer(cuda, checked, world, mode, cfg):
    B = 9
    kw = dict(world_x=world[0], world_y=world[1], world_z=world[2], render_width=32, render_height=32, obs_dtype=mode,
              ground_height=WORLDS[world], max_steps=128)
    g = GpuEnv(cuda, B, numerics="ieee", debug=False, checked=checked, **kw)
    if (world[0] * world[1] * world[2]) % 16:
        cfg = (0,) + cfg[1:]  # the launch stages these by itself
    f = capi.FusedConfig(*cfg)
    capi.check(g.L.mc_env_set_fused_config(g.h, ctypes.byref(f)), "set_fused_config", L=g.L)
    o = O.OracleEnv(batch_size=B, **kw)
    assert (o.voxels[:, -1] >= 0).any()
    g.reset()
    o.reset()
    d = diff_report(g.state(), oracle_state(o))
    assert not d, f"reset: {d}"
    rng = np.random.default_rng(71)
    for s in range(8):
        btn = np.zeros((B, 8), np.int8)
        btn[:, 4] = 1  # jump
        look = np.stack([rng.uniform(-0.8, 0.8, B), rng.uniform(-0.1, 0.5, B)], 1).astype(np.float32)
        g.step(btn, look, capi.FORM_FUSED)
        o.step(btn, look)
        d = diff_report(g.state(), oracle_state(o))
        assert not d, f"step {s}: {d}"
    if checked:
        out = (ctypes.c_int32 * 4)()
        capi.check(g.L.mc_debug_bounds_report(capi.NUMERICS_IEEE, out, None), "bounds report", L=g.L)
        assert list(out) == [0, 0, 0, 0]
    capi.check(g.L.mc_env_check_error(g.h, None), "check_error", L=g.L)
    g.close()
