"""Steps and resets of images of a few thousand pixels a row, with the default launch shape, against the CPU oracle."""
import pytest

import test_images_gpu as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["uint8", "uint8_minimal", "float32"])
@pytest.mark.parametrize("res", [(2401, 5), (3000, 2), (4400, 7)])
def test_wide_images(cuda, mode, res):
    T.run(cuda, 2, 4, 101, res=res, obs_dtype=mode, episode_length=3, regen="per_env")
    T.run(cuda, 1, 3, 102, world=(32, 32, 32), res=res, obs_dtype=mode, episode_length=2)
