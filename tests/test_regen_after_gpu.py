"""Steps of launches without the images' common path, whose worlds a kernel after
the images regenerates: both rules, alone and as groups of a ragged batch beside
one that regenerates its own."""
import pytest

import test_images_gpu as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("regen", ["all", "per_env"])
@pytest.mark.parametrize("world, res, cfg", [((70, 16, 66), (24, 20), None), ((64, 64, 64), (16, 16), None),
                                             ((25, 22, 39), (24, 24), None),
                                             ((16, 16, 16), (32, 32), (0, 8, 4, 4, 1, 0)),
                                             ((32, 32, 32), (32, 32), (0, 8, 3, 8, 4, 1))])
def test_worlds_regenerated_after_the_images(cuda, regen, world, res, cfg):
    T.run(cuda, 7, 9, 111, world=world, res=res, regen=regen, cfg=cfg, obs_dtype="uint8", episode_length=3)
    for B in (48, 49, 70):  # by the images, and by the kernel after them
        T.run(cuda, B, 5, 112, world=world, res=(8, 8), regen=regen, cfg=cfg, obs_dtype="uint8_minimal", episode_length=4)


@pytest.mark.parametrize("regen", ["all", "per_env"])
def test_groups_with_and_without_a_common_path(cuda, regen):
    import torch
    from minecu import MineEnv, _C
    from minecu.ragged import RaggedBatch
    groups = [(33, (16, 16, 16), 32, 4), (53, (70, 16, 70), 24, 3), (60, (25, 22, 39), 24, 4), (9, (64, 64, 64), 16, 5), (21, (8, 8, 8), 16, None)]

    def make():
        return [MineEnv(batch_size=b, world_x=w[0], world_y=w[1], world_z=w[2], render_width=r, render_height=r,
                        ground_height=min(8, w[1] // 2), obs_dtype="uint8", episode_length=el, regen=regen, device=cuda)
                for b, w, r, el in groups]

    ra, sb = make(), make()
    batch = RaggedBatch(ra)
    batch.reset()
    for e in sb:
        e.reset()
        e.form = "plain"
    acts = torch.empty((13, batch.total), dtype=torch.uint8, device=cuda)
    _C.philox_actions(acts, 0, 0, 41, True)
    for s in range(13):
        out = batch.step(acts[s])
        for gi, (e, (_, _, d)) in enumerate(zip(sb, out)):
            _, _, dones = e.step(acts[s, batch.group_slice(gi)])
            torch.cuda.synchronize()
            assert torch.equal(d, dones)
            for k in ("voxels", "positions", "obs_buffer", "rewards", "do_reset", "step_count"):
                x, y = getattr(ra[gi], k), getattr(e, k)
                if x.dtype == torch.float32:
                    x, y = x.view(torch.int32), y.view(torch.int32)
                assert torch.equal(x, y), f"step {s} group {gi} {k}"
    batch.check_error()
