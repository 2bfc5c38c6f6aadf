"""The default launch shape of images of a few thousand pixels a row: one exists
wherever some team's bands fit a CTA's shared memory (host arithmetic, no GPU)."""
import ctypes

import pytest

from minecu import capi


def default_shape(B, W, H, world, mode):
    c = capi.make_config(B, *world, W, H, obs_dtype=mode)
    f, smem = capi.FusedConfig(), ctypes.c_int64(-1)
    rc = capi.lib().mc_default_fused_config(ctypes.byref(c), 148, 1, ctypes.byref(f), ctypes.byref(smem))
    return rc, f, smem.value


@pytest.mark.parametrize("world", [(16, 16, 16), (32, 32, 32), (9, 13, 11), (48, 48, 48)],
                         ids=lambda w: "x".join(map(str, w)))
@pytest.mark.parametrize("mode", ["uint8", "uint8_minimal", "float32"])
def test_wide_images_of_few_envs_have_a_shape(mode, world):
    for W in (1973, 2269, 2306, 2401, 2999, 3000, 3500, 4001, 4400):
        for H in (1, 2, 5, 64):
            for B in (1, 64):
                rc, f, smem = default_shape(B, W, H, world, mode)
                assert rc == capi.MC_OK, (B, W, H, capi.last_error())
                assert smem <= 227 * 1024 and f.warps_per_cta % f.team_warps == 0


@pytest.mark.parametrize("world", [(16, 16, 16), (32, 32, 32), (9, 13, 11)], ids=lambda w: "x".join(map(str, w)))
@pytest.mark.parametrize("mode", ["uint8", "uint8_minimal"])
def test_the_widest_images_of_a_plain_band_have_a_shape(mode, world):
    """The bytes to spare of images that start at any byte take no width away."""
    for W in range(4400, 4432):
        for H in (1, 3):
            head = 224 + 13 * 4 * 16 + 64 + (W + H) * 4 + 15 & ~15
            band = W * 4 * 3 + 15 & ~15  # 8-wide tiles: four rows
            if head + 256 + 4 * (16 + 128 + band) > 227 * 1024:
                continue  # one unstaged team of 4 warps does not fit
            for B in (1, 64, 4096):
                rc, f, smem = default_shape(B, W, H, world, mode)
                assert rc == capi.MC_OK and smem <= 227 * 1024, (B, W, H, capi.last_error())
