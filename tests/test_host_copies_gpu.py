"""Host-buffer steps through the copies: the fused form and ragged batches take
them for buffers that the kernels cannot use in place (rewards off a 4-byte
boundary), call after call through the two buffers of each direction, against
steps from device memory."""
import ctypes

import numpy as np
import pytest

from minecu import capi
import oracle as O
from mc_harness import GpuEnv, diff_report

pytestmark = pytest.mark.gpu

K = 7


def _host(torch, n, off):
    """Pinned bytes with `off` to spare in front (filled with 99)."""
    t = torch.full((n + 16,), 99, dtype=torch.uint8, pin_memory=True)
    return t, t.data_ptr() + off


@pytest.mark.parametrize("off", [0, 2])
@pytest.mark.parametrize("form", [capi.FORM_FUSED, capi.FORM_PLAIN])
def test_env_steps_through_copies(cuda, form, off):
    import torch
    B = 333
    envs = [GpuEnv(cuda, B, debug=False, episode_length=4) for _ in range(2)]
    ref, env = envs
    for g in envs:
        g.reset()
    acts = np.stack([O.philox_actions(B, s, 131, break_half=True) for s in range(K)])
    act, act_p = _host(torch, K * B, 1)
    act[1:1 + K * B] = torch.from_numpy(acts).reshape(-1)
    rew, rew_p = _host(torch, K * B * 4, off)
    done, done_p = _host(torch, K * B, 3)
    s = torch.cuda.current_stream().cuda_stream
    for k in range(K):
        capi.check(env.L.mc_env_step_host(env.h, act_p + k * B, rew_p + 4 * k * B, done_p + k * B, form, s), "step_host")
    capi.check(env.L.mc_env_host_join(env.h, s), "join")
    torch.cuda.synchronize()
    for k in range(K):
        ref.step_discrete(acts[k], form)
        st = ref.state()
        assert np.array_equal(rew[off + 4 * k * B:off + 4 * (k + 1) * B].numpy(), st["rewards"].view(np.uint8)), k
        assert np.array_equal(done[3 + k * B:3 + (k + 1) * B].numpy(), st["do_reset"]), k
    assert not diff_report(env.state(), ref.state())
    assert (rew[:off] == 99).all() and (rew[off + 4 * K * B:] == 99).all()
    for g in envs:
        g.close()


@pytest.mark.parametrize("off", [0, 2])
def test_ragged_steps_through_copies(cuda, off):
    import torch
    sizes = [(37, 16), (21, 8), (64, 16)]
    total = sum(b for b, _ in sizes)

    def make():
        return [GpuEnv(cuda, b, world_size=w, render_width=16, render_height=16, ground_height=4, debug=False,
                       episode_length=3 + i) for i, (b, w) in enumerate(sizes)]

    ref, env = make(), make()
    L = env[0].L
    r = ctypes.c_void_p()
    capi.check(L.mc_ragged_create((ctypes.c_void_p * len(env))(*[e.h for e in env]), len(env), ctypes.byref(r)), "create")
    for g in ref + env:
        g.reset()
    acts = np.stack([O.philox_actions(total, s, 132, break_half=True) for s in range(K)])
    act, act_p = _host(torch, K * total, 1)
    act[1:1 + K * total] = torch.from_numpy(acts).reshape(-1)
    rew, rew_p = _host(torch, K * total * 4, off)
    done, done_p = _host(torch, K * total, 3)
    s = torch.cuda.current_stream().cuda_stream
    for k in range(K):
        capi.check(L.mc_ragged_step_host(r, act_p + k * total, rew_p + 4 * k * total, done_p + k * total, s), "step_host")
    capi.check(L.mc_ragged_host_join(r, s), "join")
    torch.cuda.synchronize()
    at = 0
    for g, (b, _) in zip(ref, sizes):
        for k in range(K):
            g.step_discrete(acts[k, at:at + b], capi.FORM_FUSED)
            st = g.state()
            o = off + 4 * (k * total + at)
            assert np.array_equal(rew[o:o + 4 * b].numpy(), st["rewards"].view(np.uint8)), k
            o = 3 + k * total + at
            assert np.array_equal(done[o:o + b].numpy(), st["do_reset"]), k
        at += b
    for a, b in zip(env, ref):
        assert not diff_report(a.state(), b.state())
    capi.check(L.mc_ragged_destroy(r), "destroy")
    for g in ref + env:
        g.close()
