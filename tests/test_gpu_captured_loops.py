"""The captured wave loops that a context keeps: a program that renders many
sizes, or many kinds of call, in turn captures each once and not again on
every call, and a loop taken up again gives what the loop launched wave by
wave gives."""
import numpy as np
import pytest

import ymrt_b200 as Y
from ymrt_b200 import scenes

pytestmark = pytest.mark.gpu


def test_sizes_in_turn_capture_once(cornell_path, halton_perm):
    """Twelve path counts, 2^10 to 2^21 (the whole default queue): seven sizes of grids, powers of four."""
    import torch
    with Y.Context(0) as c:
        setting = Y.default_setting(spp=1, ray_depth=4)
        renders = []
        for p in range(10, 22):
            w, h = 1 << (p // 2), 1 << (p - p // 2)
            renders.append((Y.Scene(c, Y.HostScene(cornell_path, w, h), halton_perm),
                            torch.zeros((h, w, 4), device="cuda")))
        torch.cuda.synchronize()
        for turn in range(3):
            for scene, out in renders:
                scene.render(setting, 1, out=out)
            n = c.counters()
            assert n["loops_captured"] == n["loops_kept"] == 7, (turn, n)


def calls(c, scene_dir, halton_perm):
    """Kinds of call: forward passes of several sizes, media, batches of one to three jobs, small and large
    backward passes, another queue capacity. Each returns its outputs."""
    import torch
    surfaces, media = scenes.scene_path("cornell", 0, scene_dir), scenes.scene_path("volumetric", 0, scene_dir)
    plain = [Y.Scene(c, Y.HostScene(surfaces, w, h), halton_perm) for w, h in ((16, 16), (61, 40), (200, 130))]
    fog = Y.Scene(c, Y.HostScene(media, 48, 40), halton_perm)

    def frame(scene, spp, **more):
        return lambda: [scene.render(Y.default_setting(spp=spp, ray_depth=8, **more), 1)[0]]

    def batch(n):
        def run():
            outs = [torch.zeros((s.height, s.width, 4), device="cuda") for s in plain[:n]]
            torch.cuda.synchronize()
            Y.render_batch(c, [(s, Y.default_setting(spp=2, ray_depth=8), 1, o) for s, o in zip(plain, outs)])
            return [o.cpu().numpy() for o in outs]
        return run

    def backward(scene, spp):
        def run():
            render = [scene, Y.default_setting(spp=spp, ray_depth=8), 1, torch.zeros((scene.height, scene.width, 4), device="cuda")]
            record = torch.zeros((Y.path_count(render), 4), device="cuda")
            grads = torch.zeros((scene.material_params().shape[0], 4), device="cuda")
            torch.cuda.synchronize()
            Y.render_batch(c, [render], [record])
            dloss = torch.ones_like(render[3])
            torch.cuda.synchronize()
            Y.render_backward(c, [render], [record], [dloss], grads)
            return [render[3].cpu().numpy(), record.cpu().numpy(), grads.cpu().numpy()[:, :3]]
        return run

    def capacity(paths, run):
        def at():
            Y.library().ymrt_set_queue_capacity(c.h, paths)
            try:
                return run()
            finally:
                Y.library().ymrt_set_queue_capacity(c.h, 0)
        return at

    return [frame(plain[0], 1), frame(plain[1], 1), frame(plain[2], 4), frame(fog, 1, volume=True),
            frame(fog, 2, volume=True, distant_light=True), batch(1), batch(2), batch(3), backward(plain[0], 1),
            backward(plain[2], 4), backward(plain[1], 1), capacity(1 << 12, frame(plain[2], 1)), frame(plain[2], 1),
            frame(plain[0], 1, env_light=True), capacity(1 << 13, backward(plain[2], 1))]


def test_kinds_of_call_in_turn(scene_dir, halton_perm):
    """Each call of two rounds in one context against the same call in a context that captures nothing. Pixels and
    records differ by the order of their additions (at most 128, 1e-5 relative); an albedo gradient has positive
    terms (dLoss/dImage = 1), fewer than 1e6 in groups: 5e-4."""
    with Y.Context(0, graph_loop=0) as c:
        want = [run() for run in calls(c, scene_dir, halton_perm)]
        assert c.counters()["loops_captured"] == 0
    with Y.Context(0) as c:
        kinds = calls(c, scene_dir, halton_perm)
        for turn in range(2):
            for k, run in enumerate(kinds):
                for part, (g, w) in enumerate(zip(run(), want[k])):
                    rtol = 5e-4 if part == 2 else 1e-5
                    np.testing.assert_allclose(g, w, rtol=rtol, atol=1e-6, err_msg=f"turn {turn} call {k} part {part}")
        assert c.counters()["loops_kept"] <= 16
