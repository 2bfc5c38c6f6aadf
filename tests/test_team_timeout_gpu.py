"""Copies that time out in teams whose warps are not abreast: units without a
wait (buried cameras) between units with one, and, in the general pass, waits
that run out for some warps of a team and not for others.  Every warp of a team
then has to take the same turn; the results equal the CPU oracle's bit for bit.
The waits give up after a set number of polls while the copies, ordinary ones,
complete."""
import numpy as np
import pytest

from minecu import capi
import oracle as O
from mc_harness import GpuEnv, actions_for, diff_report, oracle_state

pytestmark = pytest.mark.gpu

TEAMS = {"4": (1, 8, 3, 8, 4, 1), "8": (1, 8, 3, 16, 8, 1), "4_depth2": (2, 8, 2, 8, 4, 1),
         "per_warp_4": (1, 8, 3, 8, 4, 0)}


@pytest.mark.parametrize("polls", [0, 1, 3])
@pytest.mark.parametrize("where", ["buried", "above"])
@pytest.mark.parametrize("team", sorted(TEAMS))
def test_every_warp_of_a_team_gives_up_together(cuda, team, where, polls):
    B, L = 1300, capi.lib()
    kw = dict(render_width=32, render_height=32, obs_dtype="uint8", gravity=0.0, ground_height=8, episode_length=30)
    g = GpuEnv(cuda, B, numerics="ieee", debug=False, **kw)
    g.set_fused(*TEAMS[team])
    g.set_regen(True)
    o = O.OracleEnv(batch_size=B, world_size=16, regen="per_env", **kw)
    g.reset()
    o.reset()
    rng = np.random.default_rng(91)
    pos = np.empty((B, 3), np.float32)
    pos[:, 0], pos[:, 2] = rng.uniform(2, 6, B), rng.uniform(2, 6, B)
    # eyes: in the ground and in the open, or above the world and inside it, in turn
    low, high = (4.0, 9.0) if where == "buried" else (9.0, 15.5)
    pos[:, 1] = np.where(rng.random(B) < 0.5, low, high)
    st = dict(positions=pos, pitches=np.full(B, -0.5, np.float32), yaws=rng.uniform(-3, 3, B).astype(np.float32),
              step_count=rng.integers(0, 30, B).astype(np.int32))
    g.load(st)
    for k, a in st.items():
        getattr(o, k)[...] = a
    capi.check(L.mc_env_set_wait_limit(g.h, polls), "set_wait_limit")
    for s in range(12):
        _, btn, look = actions_for(B, s, 91, 0.1, True)
        g.step(btn, look, capi.FORM_FUSED)
        o.step(btn, look)
        d = diff_report(g.state(), oracle_state(o))
        assert not d, f"step {s}: {d}"
    if polls == 0:
        assert L.mc_env_check_error(g.h, None) == capi.MC_ERR_KERNEL and "timed out" in capi.last_error()
    g.close()
