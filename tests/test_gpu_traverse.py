"""Closest hits and occlusion of the 8-wide traversal against a float64 brute
force over every triangle (instances transformed to world space), for ray
counts at the edges of warps and blocks. Rays whose float64 answer is within
1e-4 of changing (an edge, the end of the occlusion interval) are left out:
float32 coordinates of order 1 and the transforms' two roundings put a hit
less than 1e-5 away from where float64 finds it."""
import numpy as np
import pytest

import ymrt_b200 as Y
from ymrt_b200 import scenes

pytestmark = pytest.mark.gpu


def world_triangles(host):
    otw = host.transforms()[0].astype(np.float64).reshape(-1, 4, 4)
    tris, boundary, owner, index = [], [], [], []
    for k, inst in enumerate(host.instances()):
        geometry, transform, treat = int(inst[0]), int(inst[1]), int(inst[4])
        order = host.triangles(geometry).reshape(-1)
        p = host.mesh_corners(geometry)[order, :3].astype(np.float64)
        m = otw[transform]
        w = p[:, :1] * m[0, :3] + p[:, 1:2] * m[1, :3] + p[:, 2:] * m[2, :3] + m[3, :3]
        tris.append(w.reshape(-1, 3, 3))
        count = len(tris[-1])
        boundary += [treat != 0] * count
        owner += [k] * count
        index += range(count)
    return np.concatenate(tris), np.array(boundary), np.array(owner), np.array(index)


def brute_force(tri, o, d):
    """(rays, triangles): distance (inf: no hit) and the distance to an edge in barycentric units."""
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    p = np.cross(d[:, None], e2[None])
    det = (p * e1[None]).sum(-1)
    s = o[:, None] - tri[None, :, 0]
    u = (s * p).sum(-1) / det
    q = np.cross(s, e1[None])
    v = (d[:, None] * q).sum(-1) / det
    t = (e2[None] * q).sum(-1) / det
    margin = np.minimum(np.minimum(u, v), 1 - u - v)
    return np.where((margin >= 0) & (t > 1e-7), t, np.inf), np.where(t > 0, np.abs(margin), np.inf)


@pytest.mark.parametrize("scene", ["cornell", "volumetric", "glossy"])
@pytest.mark.parametrize("n", [1, 31, 33, 129, 1500])
def test_against_brute_force(ctx, scene, n, halton_perm, scene_dir):
    check(ctx, scene, n, halton_perm, scene_dir, 3)


@pytest.mark.parametrize("leaf", [1, 2, 4])
def test_leaf_sizes(ctx, leaf, halton_perm, scene_dir):
    """Leaves of one to four triangles, and of as many instances in the top level."""
    check(ctx, "volumetric", 1000, halton_perm, scene_dir, leaf)


def check(ctx, scene, n, halton_perm, scene_dir, leaf):
    host = Y.HostScene(scenes.scene_path(scene, 3, scene_dir), 64, 64, max_leaf_triangles=leaf)
    sc = Y.Scene(ctx, host, halton_perm)
    tri, boundary, owner, index = world_triangles(host)
    rng = np.random.default_rng(n)
    lo, hi = tri.min((0, 1)), tri.max((0, 1))
    o = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    t, edge = brute_force(tri, o.astype(np.float64), d.astype(np.float64))
    near = t.min(1)
    clear = (edge > 1e-4).all(1) & (near > 1e-4)
    got = sc.trace(o, d)
    hit = got["inst"] != 0xFFFFFFFF
    assert np.array_equal(hit[clear], np.isfinite(near[clear]))
    # the hit is on the nearest triangle where no other is nearly as near
    first = t.argmin(1)
    alone = clear & hit & (np.partition(t, 1, axis=1)[:, 1] > near * (1 + 1e-3) + 1e-4)
    assert np.array_equal(got["inst"][alone], owner[first][alone])
    assert np.array_equal(got["tri"][alone], index[first][alone])
    tmax = rng.uniform(0.05, 1.5, n).astype(np.float32)
    solid = np.where(boundary[None], np.inf, t)
    decided = clear & (np.abs(solid - tmax[:, None]) > 1e-4 * tmax[:, None]).all(1) & ((solid > 1e-4).all(1))
    assert np.array_equal(sc.occluded(o, d, tmax)[decided] != 0, (solid <= tmax[:, None]).any(1)[decided])
    assert n < 100 or decided.mean() > 0.5
    sc.close()
