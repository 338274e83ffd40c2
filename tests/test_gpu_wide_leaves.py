"""Leaves of more facets than a group has lanes: their facets are tested in
rounds of eight, and the first of the closest counts whichever round it is
in.

The facets of a cluster have bounding boxes about one centre (two vertices are
opposite each other, the others lie within their box), which no split
separates, so each cluster stays one leaf.  Every ray is compared with the
binary traversal, hits and misses, closest and any."""

import numpy as np
import pytest
from test_gpu_many_meshes import wall_distances
from test_gpu_wide_bvh import dot, scene_of, traverse

pytestmark = pytest.mark.gpu


def cluster(n, count, center, seed, repeats=0):
    """`count` facets about a centre of few bits; `repeats`: of the last ones
    that repeat the first."""
    rng = np.random.default_rng(seed)
    a = np.round(rng.uniform(0.1, 0.4, size=(count, n)) * 256) / 256 * rng.choice([-1.0, 1.0], size=(count, n))
    p = np.empty((count, n, n))
    p[:, 0] = a
    p[:, 1] = -a
    p[:, 2:] = a[:, None] * rng.uniform(-0.9, 0.9, size=(count, n - 2, n))
    if repeats:
        p[-repeats:] = p[:repeats]
    return (p + np.asarray(center)).astype(np.float32)


@pytest.mark.parametrize("builder", ["device", "host"])
@pytest.mark.parametrize("n", [3, 4, 5])
@pytest.mark.parametrize("counts,repeats", [((8,), 0), ((9,), 4), ((16,), 0), ((17,), 9), ((20, 7), 0), ((40, 25, 1), 12)])
def test_every_ray_equals_the_binary_traversal(painter, builder, n, counts, repeats):
    centers = [[0.5 * (k - 1)] + [0.25 * k] * (n - 1) for k in range(len(counts))]
    p = np.concatenate([cluster(n, c, centers[k], 10 * c + k, min(repeats, c // 2)) for k, c in enumerate(counts)])
    facets = np.arange(len(p) * n, dtype=np.int32).reshape(-1, n)
    desc = scene_of(n, [(p.reshape(-1, n), facets)])
    s = painter.Scene(desc, "double", False, bvh_builder=builder)
    m = s.mesh_export(0)
    sizes = sorted(int(x) for x in m["node_info"][:, 1] if x > 0)
    assert sizes == sorted(counts)
    rng = np.random.default_rng(n)
    rays = 400
    org = rng.uniform(-0.9, 0.9, size=(rays, n))
    weight = rng.dirichlet(np.ones(n) * 3, size=rays)
    at = np.einsum("rk,rkd->rd", weight, p[rng.integers(0, len(p), rays)].astype(np.float64))
    direction = np.where(np.arange(rays)[:, None] % 3 == 0, rng.normal(size=(rays, n)), at - org)
    direction[::11, 0] = 0.0
    kind, index, t, _ = s.trace(np.concatenate([org, direction], axis=1))
    anything = s.trace(np.concatenate([org, direction], axis=1), any_hit=True)
    d = direction / np.sqrt(dot(direction, direction))[:, None]
    walls = wall_distances(desc, org, d)
    found = set()
    for r in range(rays):
        best, f = traverse(m, org[r], d[r], float(walls[r]))
        assert anything[r] == (best < np.inf)
        if f >= 0:
            found.add(f)
            assert (kind[r], index[r], t[r]) == (3, f, best)
        else:
            assert kind[r] == (1 if best < np.inf else 0)
    assert len(found) >= min(8, len(p) // 2)
    s.close()
