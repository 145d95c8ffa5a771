"""The shading kernels work block by block (128 to 512 threads, stages between
barriers): renders whose waves end inside a block, at its edge and one path
past it equal the render made in one wave. The paths are the same, so pixels
differ only by the order of their additions: at most 4 shadow rays at each of
16 vertices, 64 float additions, 64 * 2^-24 < 1e-5 relative."""
import numpy as np
import pytest

import ymrt_b200 as Y
from ymrt_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene,media", [("cornell", False), ("imaged", False), ("spheres", True),
                                         ("volumetric", True), ("textured", True)])
def test_waves_ending_inside_a_block(scene, media, halton_perm, scene_dir):
    host = Y.HostScene(scenes.scene_path(scene, 0, scene_dir), 40, 24)
    setting = Y.default_setting(spp=1, ray_depth=8, volume=media, distant_light=True)
    images = {}
    for capacity in (0, 127, 128, 129, 511, 512, 513):
        with Y.Context(0, queue_capacity=capacity) as c:
            image, stats = Y.Scene(c, host, halton_perm).render(setting, 1)
            assert stats.device_errors == 0
            images[capacity] = (image, stats.extension_rays, stats.shadow_rays)
    want, rays, shadows = images.pop(0)
    assert want[..., :3].max() > 0
    for capacity, (image, r, s) in images.items():
        assert (r, s) == (rays, shadows), capacity
        np.testing.assert_allclose(image, want, rtol=1e-5, atol=1e-7, err_msg=str(capacity))
