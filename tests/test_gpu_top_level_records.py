"""What the traversal reads of the top level (a record per leaf slot, and per
node which children lead to boundary instances and which to others) after a
device rebuild equals, byte for byte, what the host makes of the same edit:
for node counts below and above the 1024 nodes that the rebuild takes at a time."""
import time

import numpy as np
import pytest

import ymrt_b200 as Y

pytestmark = pytest.mark.gpu


def many_instances(path, n, seed, max_leaf):
    """The scene's instances and n small copies of its last one, every third or so a boundary."""
    base = Y.HostScene(path, 32, 32)
    geometries = []
    for g in range(len(base.geometries())):
        c = base.mesh_corners(g)
        k = np.arange(len(c), dtype=np.uint32)
        geometries.append({"triangles": base.triangles(g), "position_indices": k, "positions": c[:, :3],
                           "normal_indices": k, "normals": c[:, 3:6]})
    inst = base.instances()
    words = np.zeros((len(inst), 8), np.uint32)
    words[:, 0], words[:, 1], words[:, 2] = inst[:, 0], inst[:, 1], 1
    words[:, 3], words[:, 4], words[:, 5] = inst[:, 2], inst[:, 3], inst[:, 4]
    own = base.transforms()[0].reshape(-1, 16)
    rng = np.random.default_rng(seed)
    m = np.tile(np.eye(4, dtype=np.float32).reshape(1, 16), (n, 1))
    m[:, 0] = m[:, 5] = m[:, 10] = 0.02
    m[:, 12:15] = rng.uniform(-0.9, 0.9, (n, 3))
    copies = np.tile(words[-1:], (n, 1))
    copies[:, 1] = len(own) + np.arange(n)
    copies[:, 5] = rng.random(n) < 0.3
    cam = base.camera()
    host = Y.HostScene.from_arrays(32, 32, np.concatenate([own, m]), geometries, np.concatenate([words, copies]),
                                   base.records("materials"), (cam[:3], (0.0, 0.0, 0.0), 40.0),
                                   max_leaf_triangles=max_leaf)
    return host, len(own), m


@pytest.mark.parametrize("n,max_leaf", [(1, 3), (9, 1), (900, 1), (1100, 1), (1100, 4), (2600, 3), (20000, 1),
                                        (20000, 3)])
def test_device_rebuild_equals_host(ctx, cornell_path, halton_perm, n, max_leaf):
    host, first, m = many_instances(cornell_path, n, n, max_leaf)
    dev = Y.Scene(ctx, host, halton_perm)
    count = min(n, 5)
    for step in range(2):
        edit = m[:count].copy()
        edit[:, 12:15] *= -0.5 - step
        t = time.perf_counter()
        dev.set_transforms(first, edit)
        t = time.perf_counter() - t
        host.set_transforms(first, edit)
        fresh = Y.Scene(ctx, host, halton_perm)
        for part in ("tlas_nodes", "tlas_prims", "instances", "tlas_kinds", "instance_slots"):
            a, b = dev.download(part), fresh.download(part)
            assert a.shape == b.shape and np.array_equal(a, b), f"edit {step}: {part}"
        kinds = dev.download("tlas_kinds")
        boundary = int((dev.download("instances").reshape(-1, 8)[:, 5] != 0).sum())
        assert bool(kinds[0] & 0xFF) == (boundary > 0) and kinds[0] >> 8
        fresh.close()
    print(f"{n} instances, {len(kinds)} nodes: device edit {t * 1e3:.2f} ms")
    dev.close()
