"""Worlds regenerated at any byte offset and of any length: the whole template,
and not a byte beside it (a view with guard bytes around and between nothing)."""
import ctypes

import numpy as np
import pytest

from minecu import capi
from mc_harness import GpuEnv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1, 2, 3, 4, 13])
@pytest.mark.parametrize("world", [(5, 5, 5), (3, 7, 5), (2, 4, 6), (9, 40, 13), (16, 16, 16), (7, 11, 23)],
                         ids=lambda w: "x".join(map(str, w)))
@pytest.mark.parametrize("cfg", [(0, 8, 4, 4, 1, 0), (0, 8, 3, 8, 4, 1)], ids=["per_warp", "team"])
def test_regenerated_worlds_hold_the_template(cuda, world, off, cfg):
    import torch
    B, n = 11, world[0] * world[1] * world[2]
    g = GpuEnv(cuda, B, world_x=world[0], world_y=world[1], world_z=world[2], render_width=8, render_height=8,
               ground_height=2, debug=False, episode_length=1)
    g.set_regen(True)
    want = g.t["voxels"][0].cpu().numpy().reshape(-1)  # one generated world
    base = torch.full((B * n + 64,), 77, dtype=torch.int8, device=cuda)
    at = 32 + off
    base[at:at + B * n] = torch.randint(0, 12, (B * n,), dtype=torch.int8, device=cuda)
    g.st.voxels = base.data_ptr() + at
    capi.check(g.L.mc_env_set_state(g.h, ctypes.byref(g.st)), "set_state")
    g.set_fused(*cfg)
    before = base.cpu().numpy()
    done = np.arange(B) % 3 != 1
    g.load(dict(step_count=np.where(done, 5, 0).astype(np.int32), positions=np.full((B, 3), 50.0, np.float32)))
    g.step(np.zeros((B, 8), np.int8), np.zeros((B, 2), np.float32), capi.FORM_FUSED)
    after = base.cpu().numpy()
    for e in range(B):
        s = slice(at + e * n, at + (e + 1) * n)
        assert np.array_equal(after[s], want if done[e] else before[s]), e
    assert (after[:at] == 77).all() and (after[at + B * n:] == 77).all()
    g.close()
