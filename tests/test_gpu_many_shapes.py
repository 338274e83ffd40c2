"""Path tracing in scenes of many flat and solid shapes, which a ray's group
tests eight at a time from 128 on: the same samples, bit for bit, as with the
same shapes but those that no ray can reach.

The others stand far behind a side wall; what leaves the box through its open
side goes away from them.  Sizes: the last below the rule, the first above it,
and rounds of eight that end early."""

import numpy as np
import pytest

from math_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,size,spectrum", [(3, [24, 20], False), (4, [6, 5, 7], True), (5, [4, 3, 4, 5], False)])
@pytest.mark.parametrize("total", [127, 128, 133, 300])
def test_samples_do_not_depend_on_shapes_out_of_reach(painter, n, size, spectrum, total):
    rng = np.random.default_rng(n)
    desc = scenes.mixed_scene(n, 60, size, 1)

    def solid(at, edge):
        return {"type": "parallelotope", "metalness": 0.0, "roughness": 0.4, "color": [0.5] * 3, "alpha": 1.0,
                "org": at, "vectors": np.eye(n) * edge}

    desc["shapes"] += [solid(rng.uniform(-0.8, 0.5, n), 0.2) for _ in range(25)]
    reached = len(desc["shapes"])
    far = []
    for k in range(total - reached + 1):  # the mesh is counted in `reached` only
        at = np.zeros(n)
        at[0] = 50.0 + k
        far.append(solid(at, 0.01))
    seen = []
    for shapes in (desc["shapes"], far[: len(far) // 2] + desc["shapes"] + far[len(far) // 2:]):
        d = dict(desc, shapes=shapes)
        if shapes is not desc["shapes"]:
            d["lights"] = [dict(x, shape=x["shape"] + len(far) // 2) for x in desc["lights"]]
        s = painter.Scene(d, "double", spectrum)
        p = s.painter(8, 5, seed=4, integrator="pt")
        p.run(1)
        seen.append((p.images()[0], p.samples()[1], p.statistics()["ray_count"]))
        p.close()
        s.close()
    assert np.array_equal(seen[0][1], seen[1][1])
    assert np.array_equal(seen[0][0], seen[1][0])
    assert seen[0][2] == seen[1][2]
    assert seen[0][0].max() > 0
