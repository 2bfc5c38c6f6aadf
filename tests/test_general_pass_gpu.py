"""The general pass of the image kernels with more envs than the grid has warps,
so that every warp takes several in turn: each stages its next world into the
slot that it has just marched, and regenerates a world right after the image
that shows it.  Under the static schedule (the stateless fused step) and the
dynamic one, bit for bit."""
import ctypes

import numpy as np
import pytest

from minecu import capi
import oracle as O
from mc_harness import GpuEnv, actions_for, diff_report, oracle_state

pytestmark = pytest.mark.gpu

B = 9600  # above 148 SMs x 4 CTAs x 8 warps
ABOVE = dict(gravity=0.0, ground_height=14)  # eyes that stay above a 16^3 world, its ground within reach


def _decode(B, device):
    import torch
    f = [torch.zeros(B, dtype=torch.float32, device=device) for _ in range(5)]
    b = [torch.zeros(B, dtype=torch.bool, device=device) for _ in range(3)]
    d = capi.DecodeBuffers()
    for name, t in zip(("forward_in", "strafe_in", "delta_yaw_in", "delta_pitch_in", "speed_mult"), f):
        setattr(d, name, t.data_ptr())
    for name, t in zip(("jump_in", "do_break", "do_place"), b):
        setattr(d, name, t.data_ptr())
    return d, f + b


def _stateless(g, btn, look, form, dec=None):
    g.buttons.copy_(g.torch.from_numpy(btn))
    g.look.copy_(g.torch.from_numpy(look))
    rc = g.L.mc_step_stateless(ctypes.byref(g.cfg), ctypes.byref(g.st), g.buttons.data_ptr(), g.look.data_ptr(),
                               None if dec is None else ctypes.byref(dec), form, None)
    capi.check(rc, "mc_step_stateless")
    g.torch.cuda.synchronize()


@pytest.mark.parametrize("mode", ["uint8", "float32", "uint8_minimal", "uint8_prebasis", "uint8_prebasis_full",
                                  "uint8_fp16", "uint8_fast"])
@pytest.mark.parametrize("kw", [ABOVE, dict()], ids=["above", "inside"])
@pytest.mark.parametrize("n, res", [(B, 8), (300, 32), (5, 33)])  # several envs a warp; images in slices
def test_stateless_fused_step_equals_the_plain_one(cuda, mode, kw, n, res):
    import torch
    envs = [GpuEnv(cuda, n, render_width=res, render_height=res, obs_dtype=mode, numerics="ieee", debug=False,
                   episode_length=5, **kw) for _ in range(2)]
    plain, fused = envs
    dec, keep = _decode(n, cuda)
    rng = np.random.default_rng(81)
    for g in envs:
        g.reset()
        g.t["pitches"].fill_(-1.4)  # down, into the world
        g.t["positions"][::3, 1] -= 4.0  # some lower than the others
        torch.cuda.synchronize()
    for s in range(6):
        _, btn, look = actions_for(n, s, 81, 0.1, True)
        btn[:, 6] = rng.random(n) < 0.1
        done = rng.random(n) < 0.1
        for g in envs:
            if mode != "uint8_prebasis_full":
                g.t["do_reset"].copy_(torch.from_numpy(done))
        _stateless(plain, btn, look, capi.FORM_PLAIN, dec)
        _stateless(fused, btn, look, capi.FORM_FUSED)
        d = diff_report(fused.state(), plain.state())
        assert not d, f"step {s}: {d}"
    del keep
    for g in envs:
        g.close()


@pytest.mark.parametrize("regen", ["all", "per_env"])
@pytest.mark.parametrize("cfg", [(1, 8, 4, 4, 1, 0), (0, 8, 4, 4, 1, 0), (1, 8, 3, 8, 4, 1)],
                         ids=["staged", "unstaged", "team"])
def test_worlds_regenerated_by_the_general_pass(cuda, regen, cfg):
    n = B if cfg[4] == 1 else 1500
    g = GpuEnv(cuda, n, render_width=8, render_height=8, numerics="ieee", debug=False, episode_length=4, **ABOVE)
    g.set_fused(*cfg)
    g.set_regen(regen == "per_env")
    o = O.OracleEnv(batch_size=n, world_size=16, render_width=8, render_height=8, obs_dtype="uint8", episode_length=4,
                    regen=regen, **ABOVE)
    g.reset()
    o.reset()
    rng = np.random.default_rng(82)
    count = rng.integers(0, 4, n).astype(np.int32)
    g.load(dict(step_count=count, pitches=np.full(n, -1.4, np.float32)))
    o.step_count[...] = count
    o.pitches[...] = np.float32(-1.4)
    for s in range(9):
        _, btn, look = actions_for(n, s, 82, 0.1, True)
        look[:, 1] -= 0.4  # eyes come back level from a reset
        g.step(btn, look, capi.FORM_FUSED)
        o.step(btn, look)
        d = diff_report(g.state(), oracle_state(o))
        assert not d, f"step {s}: {d}"
    g.check_error()
    g.close()


def test_the_stateless_fused_step_allocates_nothing(cuda):
    """Under capture it leaves kernels only, and its graph can be instantiated
    more than once at a time, as one with allocations cannot."""
    import torch
    from cuda.bindings import runtime as rt

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r[0]
        return r[1] if len(r) == 2 else r[1:]

    n = 300
    envs = [GpuEnv(cuda, n, obs_dtype="uint8", numerics="ieee", debug=False) for _ in range(2)]
    want, g = envs
    for e in envs:
        e.reset()
        e.t["do_reset"].zero_()
    _, btn, look = actions_for(n, 0, 83, 0.1, True)
    _stateless(g, btn, look, capi.FORM_FUSED)  # first use
    _stateless(want, btn, look, capi.FORM_FUSED)
    s = torch.cuda.Stream(device=cuda)
    torch.cuda.synchronize()
    ok(rt.cudaStreamBeginCapture(s.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal) + (None,))
    rc = g.L.mc_step_stateless(ctypes.byref(g.cfg), ctypes.byref(g.st), g.buttons.data_ptr(), g.look.data_ptr(), None,
                               capi.FORM_FUSED, s.cuda_stream)
    graph = ok(rt.cudaStreamEndCapture(s.cuda_stream))
    capi.check(rc, "captured step")
    execs = [ok(rt.cudaGraphInstantiate(graph, 0)) for _ in range(2)]
    for x in execs:
        ok(rt.cudaGraphLaunch(x, s.cuda_stream) + (None,))
        _stateless(want, btn, look, capi.FORM_FUSED)
    torch.cuda.synchronize()
    d = diff_report(g.state(), want.state())
    assert not d, d
    for x in execs:
        ok(rt.cudaGraphExecDestroy(x) + (None,))
    ok(rt.cudaGraphDestroy(graph) + (None,))
    for e in envs:
        e.close()
