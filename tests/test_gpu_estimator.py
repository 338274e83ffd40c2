"""The RGB estimator's images against the sets of weighted samples they stand
for: of all samples that reach a pixel the two lowest and two highest are held
out, colours by weighted luminance and background samples by weight
(src/painter/pixels/samples/create.cpp:147-250, merge.cpp:78-223), and the two
kinds' held-out samples are weighed against each other when the pixel is
resolved (merge_color.cpp:45-177).

The samples and their places are the painter's own; everything after them is
formed here from the definition, in double precision, with the weights rounded
to float.  Which of several equally bright samples is held out follows no
definition but the order of the merges; only black samples are (weighted
luminance 0), so a pixel may lie between what the heaviest and the lightest of
them give.

Tolerances: a float weight, its product with a float colour and the rounded
quotient are 4 units of 2^-24; float sums add a unit per term in the
numerator and in the denominator, of at most 256 terms to a group and eight to
each merge.  In single precision a filter factor is the difference of two
exponentials up to 1, each within two units, so a weight is off by up to three
units of 1 per axis, however small it is."""

import numpy as np
import pytest

from math_b200 import scenes
from oracle import port

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -24


def open_scene(n, size):
    """A ceiling light, a floor and a mesh, and background between them."""
    desc = scenes.mixed_scene(n, 40, size, 3)
    light = desc["lights"][0]
    floor = [s for s in desc["shapes"] if s["type"] != "mesh" and s["org"][1] == -1
             and np.all(np.array(s["vectors"])[:, 1] == 0)]
    assert len(floor) == 1
    desc["shapes"] = [desc["shapes"][light["shape"]], floor[0], desc["shapes"][-1]]
    light["shape"] = 0
    return desc


def coordinates(p, size):
    c = []
    for s in size:
        c.append(p % s)
        p //= s
    return np.array(c)


def gather(t, size, points):
    """(source pixel, sample, float weight) of the samples that reach t."""
    at = coordinates(t, size)
    stride = np.cumprod([1] + list(size[:-1]))
    out = []
    for k in range(3 ** len(size)):
        step = np.array([k // 3 ** d % 3 - 1 for d in range(len(size))])
        src = at + step
        if np.any(src < 0) or np.any(src >= size):
            continue
        p = int(src @ stride)
        w = port.gaussian_filter_weight((at - src) + 0.5 - points[p]).astype(np.float32)
        out += [(p, j, w[j]) for j in np.flatnonzero(w > 0)]
    return out


def held(order):
    return list(order) if len(order) <= 4 else list(order[:2]) + list(order[-2:])


def resolve(a, b):
    """Indices of the held-out colours (ascending keys a) and background
    samples (all of key 0) that the resolved pixel leaves out."""
    b = [0.0] * b
    ai = bi = i = 0
    while i < 2 and (ai < len(a) or bi < len(b)):
        if bi == len(b) or (ai < len(a) and a[ai] < b[bi]):
            ai += 1
        else:
            bi += 1
        i += 1
    aj, bj, i = len(a), len(b), 0
    while i < 2 and (aj > ai or bj > bi):
        if bj == bi or (aj > ai and a[aj - 1] > b[bj - 1]):
            aj -= 1
        else:
            bj -= 1
        i += 1
    return [k for k in range(len(a)) if not ai <= k < aj], [k for k in range(len(b)) if not bi <= k < bj]


def expected(t, size, points, colors, valid, off):
    """(lowest, highest) RGB of pixel t; weights may be off by `off`."""
    reach = gather(t, size, points)
    c = [(p, j, w) for p, j, w in reach if valid[p, j]]
    b = np.sort([w for p, j, w in reach if not valid[p, j]]).astype(np.float64)
    w = np.array([x[2] for x in c], np.float64)
    rgb = np.array([colors[p, j] for p, j, _ in c], np.float64).reshape(-1, 3)
    lum = np.array([port.luminance_rgb(colors[p, j]) for p, j, _ in c], np.float32)
    key = np.array([x[2] for x in c], np.float32) * lum
    order = np.argsort(key, kind="stable")
    black = np.sort(w[key == 0])
    kept_c, kept_b = held(order), held(range(len(b)))
    if len(kept_c) + len(kept_b) <= 4 and not (len(order) > 4 and not kept_b):
        return None  # too few samples to resolve the pixel
    out_c, out_b = resolve([key[k] for k in kept_c], len(kept_b))
    out = [kept_c[k] for k in out_c]
    weight_b = b.sum() - sum(b[kept_b[k]] for k in out_b)
    numerator = (w[:, None] * rgb).sum(axis=0) - sum(w[k] * rgb[k] for k in out)
    numerator_off = off * rgb.sum(axis=0)
    out_black = sum(1 for k in out if key[k] == 0)
    rest = w.sum() + weight_b - sum(w[k] for k in out if key[k] != 0)
    rest_off = off * len(reach)
    lightest = rest - black[:out_black].sum() + rest_off
    heaviest = rest - black[len(black) - out_black:].sum() - rest_off
    return (numerator - numerator_off) / lightest, (numerator + numerator_off) / heaviest


@pytest.mark.parametrize("precision,sums", [("double", "double"), ("double", "float"), ("float", "double")])
@pytest.mark.parametrize("n,size,spp,pixels", [
    (3, [9, 7], 256, 63),            # the largest group, formed and merged by two kernels
    (3, [60, 61], 256, 40),
    (3, [8, 9], 144, 72),            # one launch
    (4, [5, 6, 5], 216, 40),
    (5, [3, 4, 3, 4], 256, 20),
    (3, [300, 200], 9, 60),          # a thread per pixel
    (4, [60, 52, 53], 8, 60),
    (5, [9, 8, 9, 7], 1, 60),
    (5, [40, 40, 40, 2], 16, 40),    # ranges shorter than the last axis' stride
])
def test_images_are_those_of_the_sample_sets(painter, n, size, spp, pixels, precision, sums):
    s = painter.Scene(open_scene(n, size), precision, False)
    p = s.painter(spp, 2, seed=7, pixel_sums=sums)
    p.run(1)
    rgb, _ = p.images()
    points, colors, valid = p.samples()
    p.close()
    s.close()
    count = int(np.prod(size))
    points = points.reshape(count, spp, n - 1)
    colors = colors.reshape(count, spp, 3)
    valid = valid.reshape(count, spp).astype(bool)
    rng = np.random.default_rng(n * spp)
    unit = UNIT * (6 if sums == "double" else 6 + 2 * (256 + 8 * 3 ** (n - 1)))
    off = 3 * (n - 1) * UNIT if precision == "float" else 0.0
    seen = np.flatnonzero(valid.any(axis=1))
    checked = lit = mixed = 0
    for t in rng.choice(seen, min(pixels, len(seen)), replace=False):
        e = expected(int(t), size, points, colors, valid, off)
        if e is None:
            continue
        checked += 1
        lo, hi = e
        assert np.all(rgb.reshape(count, 3)[t] >= lo * (1 - unit) - 1e-30)
        assert np.all(rgb.reshape(count, 3)[t] <= hi * (1 + unit) + 1e-30)
        lit += hi.max() > 0
        mixed += 0 < valid[t].sum() < spp
    assert lit > 5 and checked > 10
    if spp > 16:
        assert mixed > 0  # groups of both kinds


def test_one_sample_per_pixel_takes_one_launch(painter):
    """However many pixels: carried through memory in ranges, the groups of
    1.7 million pixels took 28 launches and five times as long."""
    launches = []
    for edge in (6, 120):
        s = painter.Scene(scenes.mixed_scene(4, 40, [edge] * 3, 3), "float", False)
        p = s.painter(1, 2, seed=7)
        p.run(1)
        launches.append(p.statistics()["kernel_launches"])
        p.close()
        s.close()
    assert launches[0] == launches[1]
