"""Polygons of more than one vertex node in a batch and in the server: the nodes after the first are
found by index, which moves with the scene's place in the joint tables."""
import math

import numpy as np
import pytest

from light_garden_gb300 import abi
from light_garden_gb300.scene import Circle, ConvexPolygon, Logic, Material, Object, PointLight, pack

pytestmark = pytest.mark.gpu


def _scene(n, seed):
    r = np.random.default_rng(seed)

    def polygon():
        a = r.uniform(0, 2 * math.pi)
        return ConvexPolygon(tuple((0.2 * math.cos(a + 2 * math.pi * k / n), 0.2 * math.sin(a + 2 * math.pi * k / n))
                                   for k in range(n)), (r.uniform(-0.7, 0.7), r.uniform(-0.5, 0.5)), (0.8, 0.6))

    objects = [Object(abi.LG_OBJ_CIRCLE, Circle((r.uniform(-0.5, 0.5), 0.6), 0.15), Material(1.4)),
               Object(abi.LG_OBJ_CONVEX_POLYGON, polygon(), Material(1.5)),
               Object(abi.LG_OBJ_GEO, Logic(abi.LG_OP_AND_NOT, polygon(), Circle((0.1, 0.0), 0.1)), Material(1.3)),
               Object(abi.LG_OBJ_CONVEX_POLYGON, polygon(), None)]
    params = abi.params_default()
    params.width, params.height, params.max_bounce = 160, 120, 7
    return pack(objects, [PointLight((-0.9, -0.7), 700, (1.0, 0.9, 0.8, 1.0))], params)


SCENES = [(3, 1), (5, 2), (9, 3), (4, 4), (17, 5), (61, 6)]


def _alone(pk):
    from light_garden_gb300.runtime import Context
    with Context() as c:
        c.upload(pk)
        return c.render()[0]


@pytest.mark.parametrize("precision", [abi.LG_PRECISION_EXACT, abi.LG_PRECISION_FAST])
def test_batch(ctx, precision):
    scenes = [_scene(*s) for s in SCENES]
    for pk in scenes:
        pk.params.precision = precision
    ctx.batch_upload(scenes)
    imgs, _ = ctx.batch_render()
    for s, pk, img in zip(SCENES, scenes, imgs):
        assert np.array_equal(img, _alone(pk)), s


def test_server(ctx):
    scenes = [_scene(*s) for s in SCENES]
    ctx.serve_begin(hbm_budget_bytes=1 << 30, max_slots=4)
    ids = [ctx.serve_submit(pk) for pk in scenes]
    done = {}
    for _ in range(200):
        ctx.serve_step()
        for s, i in zip(SCENES, ids):
            if s not in done:
                img = ctx.serve_poll(i)
                if img is not None:
                    done[s] = img
        if len(done) == len(SCENES):
            break
    ctx.serve_end()
    for s, pk in zip(SCENES, scenes):
        assert np.array_equal(done[s], _alone(pk)), s
