"""Scenes of several meshes: eight bounds are tested together, a lane each,
and the meshes that a ray enters are visited in their order.  Sizes: below, at
and above a round of eight, and a last round that is nearly empty.

Closest and any hits against the binary traversal of each mesh in turn, bit
for bit; renders against the same facets as one mesh."""

import numpy as np
import pytest
from test_gpu_wide_bvh import dot, scene_of, soup, traverse

from math_b200 import scenes

pytestmark = pytest.mark.gpu


def wall_distances(desc, org, d):
    """Closest wall of the open box for each ray."""
    best = np.full(len(org), np.inf)
    for s in desc["shapes"]:
        if s["type"] == "mesh":
            continue
        lo = np.array(s["org"], np.float64)
        size = np.abs(np.array(s["vectors"])).sum(axis=0)
        axis = int(np.argmin(size))
        with np.errstate(divide="ignore", invalid="ignore"):
            x = (lo[axis] - org[:, axis]) / d[:, axis]
            p = org + d * x[:, None]
        inside = (x > 0) & (x < best)
        for i in range(org.shape[1]):
            if i != axis:
                inside &= (lo[i] < p[:, i]) & (p[:, i] < lo[i] + size[i])
        best[inside] = x[inside]
    return best


@pytest.mark.parametrize("n,count", [(3, 7), (3, 8), (3, 9), (3, 17), (4, 10), (5, 9), (5, 24)])
def test_hits_equal_the_meshes_one_by_one(painter, n, count):
    rng = np.random.default_rng(100 * n + count)
    soups = []
    for k in range(count):
        p, f = soup(n, 1 + 5 * (k % 4), 100 * count + k)
        soups.append(((0.4 * p + rng.uniform(-0.5, 0.5, size=n)).astype(np.float32), f))
    soups[-1] = soups[0]  # the first mesh again: equal distances, the first counts
    desc = scene_of(n, soups)
    s = painter.Scene(desc, "double", False)
    meshes = [s.mesh_export(k) for k in range(count)]
    corners = np.concatenate([p for p, _ in soups]).astype(np.float64).reshape(-1, n, n)
    rays = 400
    weight = rng.dirichlet(np.ones(n) * 3, size=rays)
    at = np.einsum("rk,rkd->rd", weight, corners[rng.integers(0, len(corners), rays)])
    org = rng.uniform(-0.9, 0.9, size=(rays, n))
    direction = np.where(np.arange(rays)[:, None] % 4 == 0, rng.normal(size=(rays, n)), at - org)
    direction[::9, n - 1] = 0.0  # an infinite reciprocal
    kind, index, t, _ = s.trace(np.concatenate([org, direction], axis=1))
    anything = s.trace(np.concatenate([org, direction], axis=1), any_hit=True)
    d = direction / np.sqrt(dot(direction, direction))[:, None]
    walls = wall_distances(desc, org, d)
    hits = set()
    for r in range(rays):
        best, found, base = float(walls[r]), -1, 0
        for k, m in enumerate(meshes):
            best, f = traverse(m, org[r], d[r], best)
            if f >= 0:
                found, hit_mesh = base + f, k
            base += len(m["planes"])
        assert anything[r] == (best < np.inf)
        if found >= 0:
            hits.add(hit_mesh)
            assert (kind[r], index[r], t[r]) == (3, found, best)
        else:
            assert kind[r] == (1 if best < np.inf else 0)
    assert 0 in hits and count - 1 not in hits and len(hits) > count // 2
    s.close()


@pytest.mark.parametrize("integrator", ["bpt", "pt"])
@pytest.mark.parametrize("n,size,count", [(3, [24, 20], 20), (4, [6, 5, 7], 9)])
def test_renders_equal_those_of_one_mesh(painter, n, size, count, integrator):
    rng = np.random.default_rng(n)
    desc = scenes.mixed_scene(n, 40, size, 1)
    o = desc["shapes"].pop()["objects"][0]
    objects = [dict(o, matrix=scenes.transform_matrix(n, 0.2, list(rng.uniform(-0.7, 0.7, n)))) for _ in range(count)]
    seen = []
    for meshes in ([objects], [[x] for x in objects]):
        shapes = desc["shapes"] + [{"type": "mesh", "objects": m} for m in meshes]
        s = painter.Scene(dict(desc, shapes=shapes), "double", False)
        p = s.painter(8, 5, seed=4, integrator=integrator)
        p.run(1)
        seen.append((p.images()[0], p.samples()[1]))
        p.close()
        s.close()
    assert np.array_equal(seen[0][1], seen[1][1])
    assert np.array_equal(seen[0][0], seen[1][0])
    assert seen[0][0].max() > 0
