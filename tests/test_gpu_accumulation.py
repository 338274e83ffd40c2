"""RGB accumulation: the two ways a pass's samples reach the pixels (one
launch for small screens, groups and a merge for larger ones) and the ranges
a large screen is split into.

A screen too large for the single launch is compared, bit for bit, with its
slabs, which are small enough for it; the single launch on small screens is
held to the reference's estimator by the parity tests.
"""

import numpy as np
import pytest

from math_b200 import scenes

pytestmark = pytest.mark.gpu


def slabs_equal_the_screen(painter, n, edge, rows, spp, precision, sums, step):
    desc = scenes.mixed_scene(n, 60, [edge] * (n - 2) + [rows], 3)
    s = painter.Scene(desc, precision, False)
    whole = s.painter(spp, 2, seed=5, pixel_sums=sums)
    whole.run(2)
    rgb, rgba = whole.images()
    whole.close()
    assert np.isfinite(rgb).all() and rgb.max() > 0
    row = edge ** (n - 2)
    for begin in range(0, rows, step):
        end = min(rows, begin + step)
        p = s.painter(spp, 2, seed=5, pixel_sums=sums, slab=(begin, end))
        p.run(2)
        a, b = p.images()
        p.close()
        assert np.array_equal(a, rgb[begin * row:end * row])
        assert np.array_equal(b, rgba[begin * row:end * row])
    s.close()


@pytest.mark.parametrize("precision,sums", [("float", "double"), ("double", "float")])
@pytest.mark.parametrize("n,edge,rows,spp,step", [
    (3, 61, 67, 1, 33),    # a group of one sample
    (3, 50, 61, 9, 40),    # nine samples: the smallest partial selection
    (3, 47, 64, 64, 31),
    (3, 46, 47, 256, 11),  # the largest group
    (4, 11, 13, 8, 4),
    (4, 9, 17, 27, 3),
    (5, 5, 7, 16, 3),
    (5, 4, 11, 81, 2),
])
def test_slabs_equal_the_screen(painter, n, edge, rows, spp, step, precision, sums):
    slabs_equal_the_screen(painter, n, edge, rows, spp, precision, sums, step)


def test_a_screen_of_several_ranges(painter):
    """5-space, 50,625 pixels: more groups than the scratch holds at once."""
    slabs_equal_the_screen(painter, 5, 15, 15, 1, "float", "double", 5)
