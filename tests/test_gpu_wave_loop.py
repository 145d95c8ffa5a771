"""The captured wave loop (shadow rays of a wave traced beside the next wave,
continuing rays grouped from 131,072 up) against the loop launched wave by
wave without grouping: the same paths, so the same ray counts, and pixels that
differ only by the order of their additions (at most 4 shadow rays at each of
8 vertices a sample, 4 samples: 128 additions, 128 * 2^-24 < 1e-5 relative)."""
import numpy as np
import pytest

import ymrt_b200 as Y

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,spp", [(16, 16, 1), (64, 40, 4), (361, 363, 1), (640, 480, 4)])
def test_captured_loop_equals_waves(cornell_path, halton_perm, width, height, spp):
    host = Y.HostScene(cornell_path, width, height)
    setting = Y.default_setting(spp=spp, ray_depth=8)
    with Y.Context(0, graph_loop=0, sort_rays=0) as c:
        want, st = Y.Scene(c, host, halton_perm).render(setting, 2)
    with Y.Context(0) as c:
        scene = Y.Scene(c, host, halton_perm)
        for _ in range(2):  # the second render runs the captured loop again
            got, sg = scene.render(setting, 2)
            assert sg.device_errors == 0
            assert (sg.extension_rays, sg.shadow_rays) == (st.extension_rays, st.shadow_rays)
            np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("n_scenes", [2, 3, 5])
def test_grouped_batch_equals_single_renders(scene_dir, halton_perm, n_scenes):
    """Several scenes in waves large enough to be grouped (the scene is part
    of the grouping key): each image equals its render made alone (bound as above)."""
    import torch
    from ymrt_b200 import scenes
    setting = Y.default_setting(spp=4, ray_depth=8)
    with Y.Context(0) as c:
        batch = [Y.Scene(c, Y.HostScene(scenes.scene_path("cornell", k, scene_dir), 301, 303 + k), halton_perm)
                 for k in range(n_scenes)]
        outs = [torch.zeros((s.height, s.width, 4), dtype=torch.float32, device="cuda") for s in batch]
        torch.cuda.synchronize()
        st = Y.render_batch(c, [(s, setting, 1, o) for s, o in zip(batch, outs)])
        assert st.device_errors == 0
        for s, o in zip(batch, outs):
            want, _ = s.render(setting, 1)
            np.testing.assert_allclose(o.cpu().numpy(), want, rtol=1e-5, atol=1e-7)
