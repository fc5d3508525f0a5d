"""Refraction with a cosine that the double-float Fresnel term cannot hold: below 2^-60 (a ray along a face)
and zero or nearly so (the critical angle).  The exact mode decides these in FP64; against the oracle bit
for bit, colours included."""
import math

import numpy as np
import pytest

from light_garden_gb300 import abi
from light_garden_gb300.scene import Material, Object, Rect, SpotLight, pack
from parity import exact

pytestmark = pytest.mark.gpu


def _check(oracle, objects, lights, pairs):
    from light_garden_gb300.runtime import Context

    params = abi.params_default()
    params.width, params.height, params.max_bounce, params.record_paths = 170, 100, 3, 1
    pk = pack(objects, lights, params)
    with Context(scan_pairs=pairs) as ctx:
        ctx.upload(pk)
        ctx.trace()
        segs, paths = ctx.segments(paths=True)
    o_segs, o_paths, _, _ = oracle.trace(pk)
    rep = exact(segs, paths, o_segs, o_paths)
    assert rep.ok(), rep
    return o_segs, o_paths


@pytest.mark.parametrize("pairs", [0, 16])  # a generation in one launch, in three
@pytest.mark.parametrize("exponent", [-57, -59, -60, -61, -62, -66])  # of the incidence's cosine
def test_along_a_face(gpu, oracle, exponent, pairs):
    """Rays of slope 2^exponent from the middle of a rect of index 1/2 whose half height they climb within the
    canvas; their refracted rays leave at a common angle."""
    rng = np.random.default_rng(-exponent)
    slope = 2.0 ** exponent
    objects = [Object(abi.LG_OBJ_RECT, Rect((0.0, 0.0), 2.0, slope), Material(0.5))]
    lights = [SpotLight((x, 0.0), slope, (1.0, slope), 64, (1.0, 0.8, 0.6, 1.0)) for x in rng.uniform(-0.9, 0.0, 8)]
    _, paths = _check(oracle, objects, lights, pairs)
    first = paths[(paths["gen"] == 0) & (paths["source"] == 0)]
    assert (first["hit"] == 0).sum() > 100, len(first)


@pytest.mark.parametrize("pairs", [0, 16])
@pytest.mark.parametrize("index", [2.0, 1.5, 1.0])
def test_critical_angle(gpu, oracle, index, pairs):
    """Rays out of a rect within some hundred ulp of its critical angle: the refracted cosine is 0 or a few
    2^-27.  (Index 1: along the face.)"""
    objects = [Object(abi.LG_OBJ_RECT, Rect((0.0, 0.0), 1.0, 0.5), Material(index))]
    a = math.pi / 2 - math.asin(1.0 / index) if index > 1.0 else 2.0 ** -26  # from the face
    rng = np.random.default_rng(int(10 * index))
    lights = []
    for k in range(16):
        d = a + rng.integers(-8, 9) * 2.0 ** -52
        lights.append(SpotLight((rng.uniform(-0.4, -0.2), 0.25 - 0.4 * min(a, 1.0) * rng.uniform(0.2, 0.5)), 2.0 ** -45,
                                (math.cos(d), math.sin(d)), 128, (1.0, 0.8, 0.6, 1.0)))
    _check(oracle, objects, lights, pairs)
