"""Ray queries over the wide BVH (eight children to a node, eight lanes to a
ray) against the binary traversal it stands for.

The oracle walks the exported binary nodes one ray at a time in the
reference's order (near side first, a box tested when it is reached, the
first of equally distant facets kept), in double precision with the
library's operation order, so kinds, indices and distances are compared bit
for bit.  Sizes: a root that is a leaf, trees that end above, at and below a
wide node's three levels, leaves of more than eight facets (all facets alike:
the split finds no side) and facets given twice (ties in the distance).
"""

import numpy as np
import pytest

from math_b200 import scenes

pytestmark = pytest.mark.gpu


def soup(n, count, seed, twice=False):
    """`count` small random simplices in the unit cube; `twice`: every second
    one repeats the one before it."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(-0.6, 0.6, size=(count, 1, n)) + rng.normal(size=(count, n, n)) * 0.35
    if twice:
        p[1::2] = p[0::2][: len(p[1::2])]
    return p.astype(np.float32).reshape(-1, n), np.arange(count * n, dtype=np.int32).reshape(count, n)


def scene_of(n, meshes):
    desc = scenes.mixed_scene(n, 40, [4] * (n - 1), 1)
    desc["shapes"] = [s for s in desc["shapes"] if s["type"] != "mesh"]
    for points, facets in meshes:
        desc["shapes"].append({"type": "mesh", "objects": [{
            "points": points, "facets": facets, "matrix": np.eye(n + 1).tolist(), "metalness": 0.0,
            "roughness": 0.5, "color": [0.5, 0.5, 0.5], "alpha": 1.0}]})
    return desc


def dot(a, b):
    r = a[..., 0] * b[..., 0]
    for i in range(1, a.shape[-1]):
        r = r + a[..., i] * b[..., i]
    return r


def simplex_hits(planes, org, d):
    """Hit distance of one ray with each facet record, 0 for none."""
    n = len(org)
    with np.errstate(all="ignore"):
        t = (planes[:, 0, n] - dot(planes[:, 0, :n], org)) / dot(planes[:, 0, :n], d)
        p = d * t[:, None] + org
        ok = t > 0
        total = None
        for i in range(1, n):
            bc = dot(planes[:, i, :n], p) - planes[:, i, n]
            ok &= (bc > 0) & (bc < 1)
            total = bc if total is None else total + bc
        return np.where(ok & (total < 1), t, 0.0)


def traverse(m, org, d, best):
    """The binary traversal of one mesh: (distance, facet) or (best, -1)."""
    with np.errstate(divide="ignore"):
        rec = np.where(d == 0, np.inf, 1.0 / d)
    neg = d < 0
    hits = simplex_hits(m["planes"], org, d)
    found = -1
    stack = [0]
    while stack:
        k = stack.pop()
        lo, hi = m["node_lo"][k], m["node_hi"][k]
        near = max(0.0, float(np.max((np.where(neg, hi, lo) - org) * rec)))
        far = min(best, float(np.min((np.where(neg, lo, hi) - org) * rec)))
        if far < near:
            continue
        offset, count, axis = (int(x) for x in m["node_info"][k])
        if count == 0:
            stack += [k + 1, offset] if neg[axis] else [offset, k + 1]
            continue
        for f in m["indices"][offset:offset + count]:
            if 0 < hits[f] < best:
                best, found = float(hits[f]), int(f)
    return best, found


@pytest.mark.parametrize("builder", ["device", "host"])
@pytest.mark.parametrize("n", [3, 4, 5])
@pytest.mark.parametrize("counts,twice", [((1,), False), ((2,), False), ((5, 3), False), ((9,), False),
                                          ((33, 1, 8), False), ((70,), True), ((400,), False), ((257,), True)])
def test_closest_and_any_hit_equal_the_binary_traversal(painter, builder, n, counts, twice):
    soups = [soup(n, c, 10 * c + k, twice) for k, c in enumerate(counts)]
    desc = scene_of(n, soups)
    boxed = painter.Scene(desc, "double", False, bvh_builder=builder)
    meshes = [boxed.mesh_export(k) for k in range(len(counts))]
    rng = np.random.default_rng(n)
    rays = np.concatenate([rng.uniform(-0.9, 0.9, size=(203, n)), rng.normal(size=(203, n))], axis=1)
    rays[::7, n + 1] = 0.0  # a zero direction component: an infinite reciprocal
    # and rays at points of facets, which few of the others meet in a small mesh
    corners = np.concatenate([p for p, _ in soups]).astype(np.float64).reshape(-1, n, n)
    at = corners[rng.integers(0, len(corners), 90)]
    weight = rng.dirichlet(np.ones(n) * 3, size=90)
    org = rng.uniform(-0.9, 0.9, size=(90, n))
    aimed = np.concatenate([org, np.einsum("rk,rkd->rd", weight, at) - org], axis=1)
    rays = np.concatenate([rays, aimed])
    kind, index, t, _ = boxed.trace(rays)
    anything = boxed.trace(rays, any_hit=True)
    d = rays[:, n:] / np.sqrt(dot(rays[:, n:], rays[:, n:]))[:, None]
    facet_hits = 0
    for r in range(len(rays)):
        org = rays[r, :n]
        # from inside the box, past its open side the walls decide nothing
        wall = np.inf
        for s in desc["shapes"]:
            if s["type"] != "mesh":
                axis = int(np.argmin(np.abs(np.array(s["vectors"])).sum(axis=0)))
                x = (s["org"][axis] - org[axis]) / d[r, axis] if d[r, axis] != 0 else -1.0
                p = org + d[r] * x
                lo = np.array(s["org"])
                hi = lo + np.abs(np.array(s["vectors"])).sum(axis=0)
                inside = [(lo[i] < p[i] < hi[i]) for i in range(n) if i != axis]
                if x > 0 and all(inside):
                    wall = min(wall, x)
        best, found, base = wall, -1, 0
        for m in meshes:
            best, f = traverse(m, org, d[r], best)
            found = base + f if f >= 0 else found
            base += len(m["planes"])
        assert anything[r] == (best < np.inf)
        if found >= 0:
            facet_hits += 1
            assert (kind[r], index[r]) == (3, found)
            assert t[r] == best
        else:
            assert kind[r] == (1 if wall < np.inf else 0)
    assert facet_hits > 0
    boxed.close()


def test_a_leaf_larger_than_a_node(painter):
    """Twenty facets about one centre stay one leaf: three rounds of lanes."""
    n = 3
    rng = np.random.default_rng(3)
    a = rng.normal(size=(20, 1, n)) * 0.3
    p = np.concatenate([a, -a / 2 + rng.normal(size=(20, 1, n)) * 0.0, -a / 2], axis=1)
    p[:, 1] += np.array([0.0, 0.2, 0.1])
    p[:, 2] -= np.array([0.0, 0.2, 0.1])
    desc = scene_of(n, [(p.astype(np.float32).reshape(-1, n), np.arange(60, dtype=np.int32).reshape(20, n))])
    s = painter.Scene(desc, "double", False)
    m = s.mesh_export(0)
    rays = np.concatenate([rng.uniform(-0.9, 0.9, size=(300, n)), rng.normal(size=(300, n))], axis=1)
    rays[:150, n:] = -rays[:150, :n]
    kind, index, t, _ = s.trace(rays)
    d = rays[:, n:] / np.sqrt(dot(rays[:, n:], rays[:, n:]))[:, None]
    for r in np.flatnonzero(kind == 3):
        best, f = traverse(m, rays[r, :n], d[r], np.inf)
        assert (index[r], t[r]) == (f, best)
    assert np.count_nonzero(kind == 3) > 10
    s.close()
