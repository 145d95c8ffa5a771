"""The adjoint pass shades in phases with queued shadow rays: backward passes
whose waves end inside a block, at its edge and one path past it give the
gradients of the pass made in one wave. With dLoss/dImage = 1 every term of an
albedo gradient is positive, so the order of at most 8000 float additions
(960 pixels, 8 vertices) moves the sum by less than 8000 * 2^-24 < 5e-4."""
import numpy as np
import pytest

import ymrt_b200 as Y
from ymrt_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene,media,sun", [("cornell", False, False), ("imaged", False, False),
                                             ("spheres", False, False), ("volumetric", True, True)])
def test_backward_waves_ending_inside_a_block(scene, media, sun, halton_perm, scene_dir):
    import torch
    host = Y.HostScene(scenes.scene_path(scene, 0, scene_dir), 40, 24)
    setting = Y.default_setting(spp=1, ray_depth=8, volume=media, distant_light=sun)
    got = {}
    for capacity in (0, 127, 128, 255, 256, 257, 513):
        with Y.Context(0, queue_capacity=capacity) as c:
            sc = Y.Scene(c, host, halton_perm)
            image = torch.zeros((24, 40, 4), dtype=torch.float32, device="cuda")
            render = [sc, setting, 1, image]
            record = torch.zeros((Y.path_count(render), 4), dtype=torch.float32, device="cuda")
            grads = torch.zeros((sc.material_params().shape[0], 4), dtype=torch.float32, device="cuda")
            torch.cuda.synchronize()
            f = Y.render_batch(c, [render], [record])
            b = Y.render_backward(c, [render], [record], [torch.ones_like(image)], grads)
            assert f.device_errors == 0 and b.device_errors == 0
            assert (b.extension_rays, b.shadow_rays) == (f.extension_rays, f.shadow_rays)
            got[capacity] = grads.cpu().numpy()[:, :3]
    want = got.pop(0)
    assert want.max() > 0
    for capacity, g in got.items():
        np.testing.assert_allclose(g, want, rtol=5e-4, atol=1e-6, err_msg=str(capacity))
