"""Kernels that ask for more than 48 KB of shared memory, launched by several
painters: how much a kernel may take is one value per kernel and device, so
one painter's launch must not depend on what another painter needs.

Path tracing: the traversal stacks of a block of 256 threads pass 48 KB in
double precision above 30 levels.  Accumulation: the factors and orders of a
block's source pixels (3-space double: 50,400 bytes at 225 samples per pixel,
57,344 at 256), and a small screen's groups (5-space, sums in double: 57 KB at
16 samples, 140 KB at 81)."""

import threading

import numpy as np
import pytest
from test_bvh_depth import degenerate_scene, geometric_row, host_build

from math_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(195, 80), (80, 195)])  # 64 and 33 levels
@pytest.mark.parametrize("integrator", ["pt", "bpt"])
def test_painters_of_scenes_of_different_depth(painter, counts, integrator):
    made = []
    for count in counts:
        assert host_build(*geometric_row(count))[2] == {195: 64, 80: 33}[count]
        desc, data = degenerate_scene(count)
        s = painter.Scene(desc, "double", False, mesh_data=data)
        made.append((s, s.painter(4, 5, seed=1, integrator=integrator)))
    images = []
    for _, p in made:
        p.run(1)
        assert p.statistics()["stack_overflows"] == 0
        images.append(p.images()[0])
        assert np.isfinite(images[-1]).all() and images[-1].max() > 0
    for (s, p), image in zip(made, images):
        p.close()
        alone = s.painter(4, 5, seed=1, integrator=integrator)
        alone.run(1)
        assert np.array_equal(alone.images()[0], image)
        alone.close()
        s.close()


@pytest.mark.parametrize("n,precision,spps", [
    (3, "double", (225, 256)),  # groups and a merge
    (5, "float", (16, 81)),     # one launch
])
def test_passes_from_several_threads(painter, n, precision, spps):
    """Screens of a few pixels, so that launching takes as long as rendering."""
    passes = 200
    runs = 10
    scene = painter.Scene(scenes.mixed_scene(n, 40, [2] * (n - 1), 2), precision, False)

    def make(spp):
        return scene.painter(spp, 1, seed=4, integrator="pt", pixel_sums="double")

    alone = []
    for spp in spps:
        p = make(spp)
        for _ in range(runs):
            p.run(passes)
        alone.append(p.images()[0])
        p.close()
    painters = [make(spp) for spp in spps * 6]
    errors = []
    start = threading.Barrier(len(painters))

    def render(p):
        try:
            start.wait()
            for _ in range(runs):
                p.run(passes)
        except painter.PainterError as e:
            errors.append(str(e))

    threads = [threading.Thread(target=render, args=(p,)) for p in painters]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for p, image in zip(painters, alone * 6):
        assert np.array_equal(p.images()[0], image)
        p.close()
    scene.close()
