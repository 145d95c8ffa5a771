"""Backward passes whose jobs sample shape lights, distant lights, both or
none, on surfaces and in media: the queued shadow rays are the forward
pass's, albedo gradients equal central differences (the image is a polynomial
in an albedo that no sample depends on; at a step of 0.01 its even terms
cancel and the third-order ones are below 1 %, as in the surface test with one
kind of light), and a call with jobs of different kinds gives the sum of its
jobs' gradients (dLoss/dImage = 1: positive terms, at most 2.5e4 of them in
each, 2.5e4 * 2^-24 = 1.5e-3)."""
import numpy as np
import pytest

import ymrt_b200 as Y

pytestmark = pytest.mark.gpu

KINDS = {"shape": (True, False), "distant": (False, True), "both": (True, True), "none": (False, False)}
W, H = 47, 33


def setting(kind, volume):
    shape, distant = KINDS[kind]
    return Y.default_setting(spp=2, ray_depth=8, shape_light=shape, distant_light=distant, volume=volume, env_light=True)


def backward(c, sc, kinds, volume):
    import torch
    renders = [[sc, setting(k, volume), 1, torch.zeros((H, W, 4), device="cuda")] for k in kinds]
    records = [torch.zeros((Y.path_count(r), 4), device="cuda") for r in renders]
    grads = torch.zeros((sc.material_params().shape[0], 4), device="cuda")
    torch.cuda.synchronize()
    f = Y.render_batch(c, renders, records)
    dloss = [torch.ones_like(r[3]) for r in renders]
    torch.cuda.synchronize()
    b = Y.render_backward(c, renders, records, dloss, grads)
    assert f.device_errors == 0 and b.device_errors == 0
    assert (b.extension_rays, b.shadow_rays) == (f.extension_rays, f.shadow_rays)
    return grads.cpu().numpy()[:, :3].astype(np.float64), b.shadow_rays


@pytest.mark.parametrize("volume", [False, True])
@pytest.mark.parametrize("kind", list(KINDS))
def test_one_kind_against_differences(ctx, volumetric_path, halton_perm, kind, volume):
    sc = Y.Scene(ctx, Y.HostScene(volumetric_path, W, H), halton_perm)
    g, shadow_rays = backward(ctx, sc, [kind], volume)
    assert (shadow_rays > 0) == (kind != "none")
    params = sc.material_params()
    checked = 0
    for m in range(params.shape[0]):
        if params[m].sum() == 0.0:
            continue  # the light material
        total = []
        for eps in (0.01, -0.01):
            p = params.copy()
            p[m, :3] += eps
            sc.set_material_params(p)
            total.append(sc.render(setting(kind, volume), 1)[0][..., :3].astype(np.float64).sum((0, 1)))
        sc.set_material_params(params)
        fd = (total[0] - total[1]) / 0.02
        for k in range(3):
            if abs(fd[k]) < 1e-3 * g.max():
                continue
            assert abs(g[m, k] - fd[k]) <= 0.01 * abs(fd[k]), (m, k, g[m, k], fd[k])
            checked += 1
    assert checked >= 3
    sc.close()


@pytest.mark.parametrize("volume", [False, True])
@pytest.mark.parametrize("kinds", [("shape", "distant"), ("none", "both", "distant"), ("none", "shape"), ("none", "none")])
def test_jobs_of_different_kinds(ctx, volumetric_path, halton_perm, kinds, volume):
    sc = Y.Scene(ctx, Y.HostScene(volumetric_path, W, H), halton_perm)
    got, _ = backward(ctx, sc, kinds, volume)
    want = sum(backward(ctx, sc, [k], volume)[0] for k in kinds)
    sc.close()
    assert want.max() > 0
    np.testing.assert_allclose(got, want, rtol=1.5e-3, atol=1e-7 * want.max())
