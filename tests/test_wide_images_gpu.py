"""Steps and resets of images of a few thousand pixels a row, with the default launch shape, against the CPU oracle."""
import pytest

import test_images_gpu as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["uint8", "uint8_minimal", "float32"])
@pytest.mark.parametrize("res", [(2401, 5), (3000, 2), (4400, 7)])
def test_wide_images(cuda, mode, res):
    T.run(cuda, 2, 4, 101, res=res, obs_dtype=mode, episode_length=3, regen="per_env")
    T.run(cuda, 1, 3, 102, world=(32, 32, 32), res=res, obs_dtype=mode, episode_length=2)


@pytest.mark.parametrize("mode", ["uint8", "uint8_minimal"])
@pytest.mark.parametrize("cfg", [(1, 8, 1, 32, 1, 0), (1, 8, 1, 32, 8, 1)], ids=["per_warp", "team"])
def test_images_as_wide_as_a_shape_holds(cuda, mode, cfg):
    """The widest image whose plain bands fit the asked shape is accepted and
    drawn, although its common path, which wants 16 bytes more a warp, is not."""
    head = 13 * 4 * 16 + 64  # tables; then u and v, colours, and per warp its words, its band and (per warp or team) a world
    world = 16 + 128 + 4096 if cfg[4] == 1 else 16 + 128

    def smem(W):
        tables = head + ((W + 2) * 4 + 213 + 15 & ~15) if cfg[4] == 1 else 224 + head + ((W + 2) * 4 + 15 & ~15) + 256 + 4096
        pad = 256 if cfg[4] == 1 else 0
        return tables + pad + 8 * (world + (W * 3 + 15 & ~15))

    W = max(w for w in range(4000, 12000) if smem(w) <= 227 * 1024 and w % 32)
    assert smem(W) + 128 > 227 * 1024
    T.run(cuda, 1, 3, 103, res=(W, 2), cfg=cfg, obs_dtype=mode, episode_length=2)
