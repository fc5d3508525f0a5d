"""Polygons against the oracle, bit for bit: vertex counts around a record's edges, either
orientation, thin and far ones, under a rotation and inside a Logic node, with rays that run
through vertices and along edges (where the FP32 side test decides nothing)."""
import math

import numpy as np
import pytest

from light_garden_gb300 import abi
from light_garden_gb300.scene import Circle, ConvexPolygon, DirectionalLight, LineSegment, Logic, Material, Object, PointLight, pack
from parity import exact

pytestmark = pytest.mark.gpu


def _polygon(n, sign, squash):
    return tuple((0.25 * math.cos(sign * 2 * math.pi * k / n), 0.25 * squash * math.sin(sign * 2 * math.pi * k / n))
                 for k in range(n))


@pytest.mark.parametrize("pairs", [0, 16])  # a generation in one launch, in three
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("n,squash", [(3, 1.0), (4, 1.0), (5, 1e-3), (8, 1.0), (9, 0.5), (17, 1.0), (40, 0.8)])
def test_polygons_match_oracle(gpu, oracle, n, squash, sign, pairs):
    from light_garden_gb300.runtime import Context

    pts = _polygon(n, sign, squash)
    objects = [
        Object(abi.LG_OBJ_CONVEX_POLYGON, ConvexPolygon(pts), Material(1.5)),
        Object(abi.LG_OBJ_CONVEX_POLYGON, ConvexPolygon(pts, (0.6, 0.3), (math.cos(0.7), math.sin(0.7))), Material(1.3)),
        Object(abi.LG_OBJ_GEO, Logic(abi.LG_OP_AND_NOT, ConvexPolygon(pts), Circle((0.1, 0.0), 0.1), (-0.6, 0.2),
                                     (math.cos(-0.4), math.sin(-0.4))), Material(1.6)),
    ]
    # 64 directions from the origin of the polygons' axes meet vertices; the beam runs along y = 0
    lights = [PointLight((-0.9, 0.0), 1024, (1.0, 0.8, 0.6, 1.0)), PointLight((0.0, 0.0), 64 * n, (0.5, 0.7, 0.9, 1.0)),
              DirectionalLight((0.4, 0.4, 1.0, 1.0), 513, LineSegment((0.9, -0.5), (0.9, 0.5)))]
    params = abi.params_default()
    params.width, params.height, params.max_bounce, params.record_paths = 211, 151, 9, 1
    pk = pack(objects, lights, params)
    with Context(scan_pairs=pairs) as ctx:
        ctx.upload(pk)
        ctx.trace()
        segs, paths = ctx.segments(paths=True)
    o_segs, o_paths, _, _ = oracle.trace(pk)
    rep = exact(segs, paths, o_segs, o_paths)
    assert rep.ok(), rep
    assert rep.segments == len(o_segs) > 2000
