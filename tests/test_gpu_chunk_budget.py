"""A render that asks for more memory for its chunk buffers than a painter
takes by itself gets it, up to a fifth of the device's memory: fewer chunks
of paths, the same image."""

import numpy as np
import pytest

from math_b200 import scenes

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def test_larger_budgets_make_fewer_chunks(painter):
    # 2.3 million paths of about 11 KB each (5-space, double precision, depth 8)
    s = painter.Scene(scenes.mixed_scene(5, 60, [13] * 4, 2), "double", False)
    launches, images = [], []
    for budget in (0, 8 * GIB, 16 * GIB, 32 * GIB):
        p = s.painter(81, 8, seed=3, chunk_budget=budget)
        p.run(1)
        launches.append(p.statistics()["kernel_launches"])
        images.append(p.images()[0])
        p.close()
        painter.release_cached_memory()
    s.close()
    assert launches[1] > launches[2] > launches[3]
    assert launches[0] == launches[2]  # by itself: 16 GiB of a B200's memory
    for image in images[1:]:
        assert np.array_equal(image, images[0])
