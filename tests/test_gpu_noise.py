"""The texture nodes' evaluation with constant inputs at hand against the
walk over the node graph: the same fBm node read directly and through a
parent that passes it on unchanged (a solid node whose two inputs are both
that node blends it with itself: black + v * (white - black) = black exactly)."""
import numpy as np
import pytest

import ymrt_b200 as Y
from ymrt_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 4097])
def test_direct_and_walked_nodes_agree(ctx, scene_dir, halton_perm, n):
    base = Y.HostScene(scenes.scene_path("volumetric", 0, scene_dir), 32, 32)
    fbm = 2
    rows = base.records("textures").copy()
    assert rows[fbm][0] == 5  # the smoke's fBm node over two constants
    parent = rows[fbm].copy()
    parent[1] = parent[2] = fbm  # both inputs: the fBm node itself
    rows = np.concatenate([rows, parent[None]])
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
    cam = base.camera()
    host = Y.HostScene.from_arrays(32, 32, base.transforms()[0], geometries, words, base.records("materials"),
                                   (cam[:3], (0.0, 0.5, 0.0), 40.0), volumes=base.records("volumes"),
                                   distant_lights=base.records("distant_lights"), textures=rows)
    sc = Y.Scene(ctx, host, halton_perm)
    p = np.random.default_rng(n).uniform(-40, 40, (n, 3)).astype(np.float32)
    p[0] = 0.0
    direct, walked = sc.density(fbm, p), sc.density(len(rows) - 1, p)
    assert np.ptp(direct) > 0 or n == 1
    assert np.array_equal(direct.view(np.uint32), walked.view(np.uint32))
    sc.close()
