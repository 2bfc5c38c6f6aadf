"""The default launch shape by the number of envs, not of tiles alone: enough envs
to give every warp or team one need no bigger teams (host arithmetic, no GPU)."""
import ctypes

import pytest

from minecu import capi


def shape(B, image, world):
    c = capi.make_config(B, world, world, world, image, image)
    f = capi.FusedConfig()
    capi.check(capi.lib().mc_default_fused_config(ctypes.byref(c), 148, 1, ctypes.byref(f), None), "default")
    return f


@pytest.mark.parametrize("B, image", [(4096, 8), (8192, 8), (32768, 8), (8192, 12), (8192, 16), (4096, 20), (4096, 32),
                                      (32768, 32)])
def test_one_warp_per_env_where_envs_are_many(B, image):
    f = shape(B, image, 16)
    assert (f.coop, f.team_warps, f.tile_w) == (0, 1, 4)


@pytest.mark.parametrize("B, image", [(1024, 12), (1024, 16), (1024, 24), (2048, 16), (2048, 32)])
def test_teams_of_four_over_small_worlds(B, image):
    f = shape(B, image, 16)
    assert (f.coop, f.team_warps) == (1, 4)


@pytest.mark.parametrize("B, image, team", [(64, 8, 8), (256, 8, 8), (256, 32, 8), (512, 64, 8), (1024, 64, 8),
                                            (1024, 8, 4), (1024, 32, 4), (2048, 16, 4), (4096, 32, 4), (8192, 8, 4),
                                            (16384, 12, 4), (4096, 64, 4)])
def test_teams_over_big_worlds(B, image, team):
    f = shape(B, image, 32)
    assert (f.coop, f.team_warps) == (1, team)


@pytest.mark.parametrize("B", [1, 64, 256, 1024, 2048])
def test_images_of_two_tiles_have_no_team(B):
    assert shape(B, 8, 16).coop == 0


@pytest.mark.parametrize("B, image, world, tile", [(1024, 32, 48, 16), (4096, 32, 48, 16), (1024, 32, 64, 16),
                                                   (1024, 8, 64, 8)])
def test_worlds_above_32_kb_take_wide_tiles_by_the_tiles(B, image, world, tile):
    f = shape(B, image, world)
    assert f.coop == 1 and f.tile_w == tile
    assert world != 64 or f.team_warps == (8 if tile == 16 else 4)
