"""The FP32 search decides a hit or a miss only where its rounding cannot change the answer, and the
rounding of a coordinate to FP32 does not shrink with the object: shapes far smaller than their
distance from the canvas centre, with rays aimed within a few roundings of where a hit becomes a miss,
against the oracle bit for bit."""
import math

import numpy as np
import pytest

from light_garden_gb300 import abi
from light_garden_gb300.scene import Circle, CubicBezier, Logic, Material, Object, Rect, SpotLight, pack
from parity import exact

pytestmark = pytest.mark.gpu

RAYS = 1536  # a spot light's
COLOR = (1.0, 0.8, 0.6, 1.0)


def _spot(o, target, spread):
    """Rays from o that pass within `spread` of target, to either side."""
    d = (target[0] - o[0], target[1] - o[1])
    return SpotLight(tuple(o), 2.0 * spread / math.hypot(*d), d, RAYS, COLOR)


def _check(oracle, objects, lights, width, height, pairs, least):
    from light_garden_gb300.runtime import Context

    params = abi.params_default()
    params.width, params.height, params.max_bounce, params.record_paths = width, height, 3, 1
    pk = pack(objects, lights, params)
    with Context(scan_pairs=pairs) as ctx:
        ctx.upload(pk)
        ctx.trace()
        segs, paths = ctx.segments(paths=True)
    o_segs, o_paths, _, _ = oracle.trace(pk)
    rep = exact(segs, paths, o_segs, o_paths)
    assert rep.ok(), rep
    hits = int(((o_paths["gen"] == 0) & (o_paths["hit"] >= 0)).sum())
    rays = RAYS * len(lights)
    assert least * rays < hits < (1.0 - least) * rays, (hits, rays)  # both sides of the edge are there


@pytest.mark.parametrize("pairs", [0, 16])  # a generation in one launch, in three
@pytest.mark.parametrize("kind", ["disc", "and"])
@pytest.mark.parametrize("width,height", [(170, 100), (1600, 100)])
@pytest.mark.parametrize("radius", [5e-5, 1e-4, 2e-4, 1e-3, 1e-2])
def test_discs_near_the_corners_grazed(gpu, oracle, radius, width, height, kind, pairs):
    rng = np.random.default_rng(int(1e6 * radius) + width)
    aspect = width / height
    objects, lights = [], []
    for k in range(10):
        c = np.array([rng.choice([-1, 1]) * rng.uniform(0.6, 0.95) * aspect, rng.choice([-1, 1]) * rng.uniform(0.5, 0.95)])
        disc = Circle(tuple(c), radius)
        if kind == "and":  # the disc again, as one leaf of two
            disc = Logic(abi.LG_OP_AND, disc, Circle((c[0] + 0.5 * radius, c[1]), 3.0 * radius))
        objects.append(Object(abi.LG_OBJ_GEO if kind == "and" else abi.LG_OBJ_CIRCLE, disc, Material(1.4)))
        dist, th = radius * rng.uniform(8.0, 90.0), rng.uniform(0.2, 1.3) + rng.integers(0, 4) * math.pi / 2
        u, n = np.array([math.cos(th), math.sin(th)]), np.array([-math.sin(th), math.cos(th)])
        # the tangent point of the ray from c - dist u
        s = radius / dist
        tangent = c + radius * (n * math.sqrt(1.0 - s * s) - u * s)
        lights.append(_spot(c - dist * u, tangent, min(3e-3 * radius, 4e-7 * (aspect + 1.0))))
    _check(oracle, objects, lights, width, height, pairs, 0.2)


@pytest.mark.parametrize("pairs", [0, 16])
@pytest.mark.parametrize("size", [2e-4, 4e-3])
def test_rects_far_off_grazed(gpu, oracle, size, pairs):
    """Rays past a corner of a small rotated rect on a wide canvas."""
    rng = np.random.default_rng(int(1e6 * size))
    objects, lights = [], []
    for k in range(10):
        c = np.array([rng.choice([-1, 1]) * rng.uniform(10.0, 15.0), rng.choice([-1, 1]) * rng.uniform(0.5, 0.95)])
        rot = rng.uniform(0.1, 1.4)
        x, y = np.array([math.cos(rot), math.sin(rot)]), np.array([-math.sin(rot), math.cos(rot)])
        objects.append(Object(abi.LG_OBJ_RECT, Rect(tuple(c), size, size, (math.cos(rot), math.sin(rot))), Material(1.4)))
        corner = c + 0.5 * size * (x + y)
        o = corner + size * rng.uniform(4.0, 40.0) * (y - x) / math.sqrt(2.0)  # across the corner's diagonal
        lights.append(_spot(o, corner, 4e-6))
    _check(oracle, objects, lights, 1600, 100, pairs, 0.2)


@pytest.mark.parametrize("pairs", [0, 16])
@pytest.mark.parametrize("side,bend", [(1e-4, 0.0), (1e-3, 0.0), (1e-3, 1e-7), (1e-3, 1e-5), (1e-2, 1e-7)])
def test_flat_mirrors_from_the_centre(gpu, oracle, side, bend, pairs):
    """Nearly straight cubic mirrors that start at the canvas centre, each seen from beside its start
    along its length, with rays past its far end."""
    rng = np.random.default_rng(int(1e6 * (side + 7 * bend)))
    objects, lights = [], []
    for k in range(10):
        a = 2.0 * math.pi * (k + rng.uniform(0.4, 0.6)) / 10
        t, n = np.array([math.cos(a), math.sin(a)]), np.array([-math.sin(a), math.cos(a)])
        length = rng.uniform(0.5, 0.95)
        pts = [t * (length * j / 3) + n * (rng.uniform(-1, 1) * bend if j else 0.0) for j in range(4)]
        objects.append(Object.new_curved_mirror(CubicBezier(tuple(tuple(p) for p in pts))))
        o = t * (2.0 * side) + n * (rng.choice([-1, 1]) * rng.uniform(0.2, 0.8) * side)  # on this side of its neighbours
        lights.append(_spot(o, pts[3], 1e-7))
    _check(oracle, objects, lights, 170, 100, pairs, 0.2)
