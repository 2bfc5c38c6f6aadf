"""Admitted jobs take the device memory that the budget counts (mc_server_job_bytes)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_a_job_takes_no_more_than_its_budgeted_bytes(cuda):
    import torch
    from minecu import capi
    from minecu.server import EnvServer
    B, kw = 1_000_000, dict(world_x=6, world_y=6, world_z=6, render_width=4, render_height=4, ground_height=3)
    cfg = capi.make_config(B, 6, 6, 6, 4, 4, ground_height=3)
    want = capi.lib().mc_server_job_bytes(ctypes.byref(cfg))
    srv = EnvServer(hbm_budget_bytes=want)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    job = srv.admit(B, **kw)
    torch.cuda.synchronize()
    took = before - torch.cuda.mem_get_info()[0]
    # the driver hands memory to its pools in steps of up to 32 MiB; anything kept
    # per env beside the state (48 bytes of render record, say) is more than that
    assert took <= want + 40_000_000, (took, want)
    srv.reset(job)
    rew, done = srv.wait(srv.submit(job, torch.zeros(B, dtype=torch.uint8)))
    assert rew.shape == (B,) and not done.any()
    srv.close()
