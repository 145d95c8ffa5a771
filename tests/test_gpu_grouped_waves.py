"""Continuing rays traced grouped (YMRT_OPT_SORT_RAYS) in waves that hold
enough of them to be grouped: the same rays through the same nodes as in
slot order (equal ray, node and triangle counts), and the same outputs up to
the order of their float additions, on surfaces, with spheres and in media,
forward and backward; the context counts the waves that were grouped."""
import numpy as np
import pytest

import ymrt_b200 as Y
from ymrt_b200 import scenes

pytestmark = pytest.mark.gpu

COUNTS = ("paths", "extension_rays", "shadow_rays", "node_visits", "triangle_tests", "shadow_node_visits")
CASES = [("instanced", False), ("volumetric", True), ("spheres", False), ("spheres", True), ("textured", True)]


def check_counts(a, b):
    for k in COUNTS:
        assert a[k] == b[k], (k, a[k], b[k])


@pytest.mark.parametrize("scene,volume", CASES)
def test_forward(scene, volume, scene_dir, halton_perm):
    """4 samples, 8 vertices, 4 shadow rays each: 128 additions a pixel, 128 * 2^-24 < 1e-5."""
    with Y.Context(0, queue_capacity=1 << 20) as c:
        sc = Y.Scene(c, Y.HostScene(scenes.scene_path(scene, 0, scene_dir), 640, 481), halton_perm)
        setting = Y.default_setting(spp=4, ray_depth=8, volume=volume)
        out = {}
        for on in (1, 0):
            c.set_option("sort_rays", on)
            img, st = sc.render(setting, 3)
            assert st.device_errors == 0
            assert (c.counters()["grouped_waves"] >= 2) if on else (c.counters()["grouped_waves"] == 0)
            out[on] = (img, st.as_dict())
        check_counts(out[1][1], out[0][1])
        np.testing.assert_allclose(out[1][0], out[0][0], rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("scene,volume", [("instanced", False), ("volumetric", True)])
def test_backward(scene, volume, scene_dir, halton_perm):
    """dLoss/dImage = 1: an albedo gradient's terms are positive, summed block by block (1e3 groups of 1e3 to 1e4
    terms), so their order moves it by less than 1.2e4 * 2^-24 < 1e-3."""
    import torch
    with Y.Context(0, queue_capacity=1 << 20) as c:
        sc = Y.Scene(c, Y.HostScene(scenes.scene_path(scene, 0, scene_dir), 640, 481), halton_perm)
        render = [sc, Y.default_setting(spp=4, ray_depth=8, volume=volume), 1, torch.zeros((481, 640, 4), device="cuda")]
        record = torch.zeros((Y.path_count(render), 4), device="cuda")
        grads = torch.zeros((sc.material_params().shape[0], 4), device="cuda")
        torch.cuda.synchronize()
        Y.render_batch(c, [render], [record])
        dloss = torch.ones_like(render[3])
        torch.cuda.synchronize()
        out = {}
        for on in (1, 0):
            c.set_option("sort_rays", on)
            st = Y.render_backward(c, [render], [record], [dloss], grads)
            assert st.device_errors == 0
            assert (c.counters()["grouped_waves"] >= 1) if on else (c.counters()["grouped_waves"] == 0)
            out[on] = (grads.cpu().numpy()[:, :3], st.as_dict())
        check_counts(out[1][1], out[0][1])
        assert out[0][0].max() > 0
        np.testing.assert_allclose(out[1][0], out[0][0], rtol=1e-3, atol=1e-6 * out[0][0].max())
