"""Rays that run along a rect's face: an error of the FP32 search in the distance to the face moves the
crossing by that distance over the sine of the angle, far beyond its tolerance at steep crossings.
Small discs that touch the face stand where the two hits are close, and the rays aim at every point of the
face.  Against the oracle bit for bit."""
import math

import numpy as np
import pytest

from light_garden_gb300 import abi
from light_garden_gb300.scene import Circle, Material, Object, Rect, SpotLight, pack
from parity import exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [0, 16])  # a generation in one launch, in three
@pytest.mark.parametrize("height", [3e-6, 3e-5, 3e-4, 3e-3])  # of the lights over the face's plane
@pytest.mark.parametrize("centre", [(0.1, 0.05), (1.2, 0.6)])
def test_rays_along_a_face(gpu, oracle, centre, height, pairs):
    from light_garden_gb300.runtime import Context

    rng = np.random.default_rng(int(1e7 * height) + int(10 * centre[0]))
    a = rng.uniform(0.2, 1.3)
    x, y = np.array([math.cos(a), math.sin(a)]), np.array([-math.sin(a), math.cos(a)])
    w, h = 0.3, 0.2
    c = np.array(centre)
    at = lambda u, v: c + x * (u * w / 2) + y * (h / 2 + v)  # along the face (-1 to 1), above it
    objects = [Object(abi.LG_OBJ_RECT, Rect(tuple(c), w, h, (math.cos(a), math.sin(a))), Material(1.5))]
    for k in range(12):
        r = 10.0 ** rng.uniform(-4.5, -2.5)
        objects.append(Object(abi.LG_OBJ_CIRCLE, Circle(tuple(at(rng.uniform(-0.9, 0.9), r)), r), Material(1.4)))
    lights = []
    for k in range(8):
        o = at(-1.0 - rng.uniform(0.1, 0.5), height * rng.uniform(0.3, 1.0))
        d0, d1 = at(-1.0, 0.0) - o, at(1.1, 0.0) - o
        t0, t1 = math.atan2(d0[1], d0[0]), math.atan2(d1[1], d1[0])
        m = 0.5 * (t0 + t1)
        lights.append(SpotLight(tuple(o), abs(t1 - t0), (math.cos(m), math.sin(m)), 1500, (1.0, 0.8, 0.6, 1.0)))
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
    first = o_paths[(o_paths["gen"] == 0) & (o_paths["source"] == 0)]
    hits = [int((first["hit"] == 0).sum()), int((first["hit"] > 0).sum())]
    assert min(hits) > 1000, hits  # the face, the discs
