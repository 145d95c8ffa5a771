"""Scratch memory that grows on demand, when growing fails (host-side
injection, ymrt_debug_fail_allocations): the old block is gone then, so a
later call that the old one would have sufficed for has to allocate anew. That
is checked on the host first (with allocations failing it returns
YMRT_ERR_OOM instead of using freed memory), and only then on the device."""
import ctypes

import numpy as np
import pytest

import ymrt_b200 as Y

pytestmark = pytest.mark.gpu

OOM = -6  # YMRT_ERR_OOM


class failing_allocations:
    def __enter__(self):
        Y.library().ymrt_debug_fail_allocations(1000)

    def __exit__(self, *exc):
        Y.library().ymrt_debug_fail_allocations(0)


def backward(ctx, scene, spp):
    import torch
    w, h = scene.width, scene.height
    render = [scene, Y.default_setting(spp=spp, ray_depth=8), 1, torch.zeros((h, w, 4), device="cuda")]
    record = torch.zeros((Y.path_count(render), 4), device="cuda")
    grads = torch.zeros((scene.material_params().shape[0], 4), device="cuda")
    torch.cuda.synchronize()
    Y.render_batch(ctx, [render], [record])
    dloss = torch.ones_like(render[3])
    torch.cuda.synchronize()
    return lambda: (Y.render_backward(ctx, [render], [record], [dloss], grads), grads.cpu().numpy().copy())[1]


def test_backward_after_a_failed_larger_one(cornell_path, halton_perm):
    with Y.Context(0) as c:
        scene = Y.Scene(c, Y.HostScene(cornell_path, 64, 48), halton_perm)
        small, large = backward(c, scene, 1), backward(c, scene, 32)
        want = small()
        for step in (large, small):  # the larger grows the vertices; the smaller then has none left
            with failing_allocations(), pytest.raises(Y.YmrtError) as e:
                step()
            assert e.value.code == OOM
        # dLoss/dImage = 1: positive terms, at most 64 * 48 pixels x 8 vertices of them, 2.5e4 * 2^-24 = 1.5e-3
        np.testing.assert_allclose(small()[:, :3], want[:, :3], rtol=1.5e-3, atol=1e-6)
        assert large()[:, :3].max() > 0


def test_queues_after_a_failed_larger_capacity(cornell_path, halton_perm):
    """A program that goes back to its old queue capacity when a larger one does not fit."""
    with Y.Context(0, queue_capacity=1 << 14) as c:
        scene = Y.Scene(c, Y.HostScene(cornell_path, 64, 48), halton_perm)
        setting = Y.default_setting(spp=4, ray_depth=8)
        want, _ = scene.render(setting, 1)
        for capacity in (1 << 16, 1 << 14):
            Y.library().ymrt_set_queue_capacity(c.h, capacity)
            with failing_allocations(), pytest.raises(Y.YmrtError) as e:
                scene.render(setting, 1)
            assert e.value.code == OOM
        got, st = scene.render(setting, 1)
        assert st.device_errors == 0
        # at most 4 shadow rays at each of 8 vertices, 4 samples: 128 additions in another order, 128 * 2^-24
        np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("failures", [1, 3, 7])
def test_backward_in_smaller_waves_when_memory_is_short(cornell_path, halton_perm, failures):
    """Room for half the vertices, an eighth, or the least there is: the pass still gives its gradients."""
    with Y.Context(0) as c:
        scene = Y.Scene(c, Y.HostScene(cornell_path, 64, 48), halton_perm)
        step = backward(c, scene, 32)  # 98,304 paths: vertices for 131,072, 65,536, ..., 1024
        Y.library().ymrt_debug_fail_allocations(failures)
        try:
            got = step()
        finally:
            Y.library().ymrt_debug_fail_allocations(0)
        want = step()
        # each wave adds a block's sums: fewer than 1e6 positive terms, in 1e3 groups of 1e3, 2e3 * 2^-24
        np.testing.assert_allclose(got[:, :3], want[:, :3], rtol=5e-4, atol=1e-6)
