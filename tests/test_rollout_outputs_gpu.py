"""A rollout's outputs may start at any byte of device memory, and lie in pinned host memory."""
import ctypes

import numpy as np
import pytest

from minecu import capi
import oracle as O
from mc_harness import GpuEnv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1, 2, 4])
@pytest.mark.parametrize("where", ["device", "pinned"])
def test_rollout_outputs_at_any_byte(cuda, off, where):
    import torch
    B, K = 37, 6
    kw = dict(batch_size=B, render_width=16, render_height=16, obs_dtype="uint8", episode_length=4)
    g = GpuEnv(cuda, numerics="ieee", debug=False, **kw)
    o = O.OracleEnv(world_size=16, **kw)
    g.reset()
    o.reset()
    acts = np.stack([O.philox_actions(B, s, 7, break_half=True) for s in range(K)])
    actions = torch.from_numpy(acts).to(cuda)
    place = dict(device=cuda) if where == "device" else dict(pin_memory=True)
    rewards = torch.full((K * B * 4 + 16,), 77, dtype=torch.uint8, **place)
    dones = torch.full((K * B + 16,), 77, dtype=torch.uint8, **place)
    capi.check(g.L.mc_env_rollout(g.h, actions.data_ptr(), K, rewards.data_ptr() + off, dones.data_ptr() + off, None),
               "rollout")
    torch.cuda.synchronize()
    rew, don = rewards.cpu().numpy(), dones.cpu().numpy()
    for s in range(K):
        btn, look = O.discrete_to_buttons(acts[s], 0.1)
        o.step(btn, look)
        at = off + s * B * 4
        assert np.array_equal(rew[at:at + B * 4].view(np.uint8), o.rewards.view(np.uint8)), s
        assert np.array_equal(don[off + s * B:off + (s + 1) * B], o.do_reset), s
    for a, n in ((rew, K * B * 4), (don, K * B)):
        assert (a[:off] == 77).all() and (a[off + n:] == 77).all()
    g.close()
