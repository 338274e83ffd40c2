"""Path tracing in scenes of nothing but a mesh: from 300,000 paths on a kernel
of its own, whose samples are those of the slabs of the same screen, which
have fewer paths.  Double precision, bit for bit; in single precision the two
kernels may round differently, and a rounding may turn a path."""

import numpy as np
import pytest

from math_b200 import scenes

pytestmark = pytest.mark.gpu


def mesh_only(n, points, size):
    desc = scenes.mixed_scene(n, points, size, 1)
    desc["shapes"] = [desc["shapes"][-1]]
    center = [0.0] * n
    center[1], center[n - 1] = 2.5, -1.0
    down = [0.0] * n
    down[1] = -1.0
    desc["lights"] = [{"type": "ball", "center": center, "direction": down, "radius": 0.8,
                       "radiance": [30.0, 30.0, 30.0]}]
    return desc


@pytest.mark.parametrize("precision", ["double", "float"])
@pytest.mark.parametrize("spectrum", [False, True])
@pytest.mark.parametrize("n,size,spp,step", [(3, [150, 140], 16, 60), (4, [24, 25, 23], 27, 9)])
def test_slabs_equal_the_screen(painter, n, size, spp, step, spectrum, precision):
    desc = mesh_only(3, 400, size) if n == 3 else scenes.sphere_4d(size=size, points=800, buckets=4)
    s = painter.Scene(desc, precision, spectrum)
    whole = s.painter(spp, 5, seed=6, integrator="pt")
    whole.run(1)
    rgb, _ = whole.images()
    _, colors, valid = whole.samples()
    assert len(colors) * colors.shape[1] >= 300_000
    assert 0 < valid.mean() < 1 and rgb.max() > 0
    row = len(rgb) // size[-1]
    for begin in range(0, size[-1], step):
        end = min(size[-1], begin + step)
        p = s.painter(spp, 5, seed=6, integrator="pt", slab=(begin, end))
        p.run(1)
        first = max(0, begin - 1) * row
        _, c, v = p.samples()
        assert len(c) * c.shape[1] < 300_000
        assert np.array_equal(v, valid[first:first + len(v)])
        if precision == "double":
            assert np.array_equal(c, colors[first:first + len(c)])
            assert np.array_equal(p.images()[0], rgb[begin * row:end * row])
        else:
            same = np.isclose(c, colors[first:first + len(c)], rtol=1e-3, atol=1e-6).all(axis=-1)
            assert same.mean() > 0.999
        p.close()
    whole.close()
    s.close()
