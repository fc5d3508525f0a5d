"""Generations visited in place and direction order against queue order.

From a number of primaries and objects on, a frame's generations visit their rays sorted by cell
of the canvas and octant of directions.  The order decides which rays share a warp, never what a
ray meets: the whole frame's trace is, path for path, that of its even and its odd primaries, each
too few to be sorted.
"""
import numpy as np
import pytest

from light_garden_gb300 import abi, workloads as W
from light_garden_gb300.runtime import Context
from test_gpu_culling import _assert_same_trace

pytestmark = pytest.mark.gpu


def _scene(kind, n, prim, precision):
    if kind == "csg":
        w = W.csg_scene(seed=n, total_rays=prim, n_objects=n, width=320, height=200, string_mod=False)
    elif kind == "mid":
        w = W.mid_scene(seed=n, rays_per_light=prim // 8, n_objects=n)
    else:
        w = W.shapes_scene(seed=n, rays_per_light=prim // 4, n_objects=n)
    w.params.width, w.params.height, w.params.max_bounce = 401, 203, 5
    w.params.precision, w.params.accum = precision, abi.LG_ACCUM_FIXED64
    pk = w.packed()
    pk.params.record_paths = 1
    return pk


def _trace(pk, stride=1, offset=0):
    pk.params.ray_stride, pk.params.ray_offset = stride, offset
    with Context(culling=abi.LG_CULL_ON) as ctx:
        ctx.upload(pk)
        ctx.trace()
        return ctx.segments(paths=True)


@pytest.mark.parametrize("precision", [abi.LG_PRECISION_EXACT, abi.LG_PRECISION_FAST])
@pytest.mark.parametrize("kind,n,prim,bounces", [("mid", 48, 65536, 6), ("csg", 192, 16384, 8), ("csg", 48, 65536, 6),
                                                 ("shapes", 96, 32768, 6), ("shapes", 24, 131072, 5)])
def test_sorted_generations_trace_the_same(gpu, kind, n, prim, bounces, precision):
    pk = _scene(kind, n, prim, precision)
    pk.params.max_bounce = bounces
    whole = _trace(pk)
    halves = [np.concatenate(x) for x in zip(_trace(pk, 2, 0), _trace(pk, 2, 1))]
    drawn = [h[halves[1]["source"] == abi.LG_SRC_TRACE] for h in halves]
    _assert_same_trace([w[whole[1]["source"] == abi.LG_SRC_TRACE] for w in whole], drawn)
    if precision == abi.LG_PRECISION_EXACT:
        key = lambda s, p: np.sort(s.view(np.dtype((np.void, s.dtype.itemsize)))[p["source"] == abi.LG_SRC_TRACE], axis=0)
        assert key(*whole).tobytes() == key(*halves).tobytes()


def _batch(ctx, packs):
    ctx.batch_upload(packs)
    return ctx.batch_render()


@pytest.mark.parametrize("count", [2, 17, 70])
def test_batch_of_many_scenes_is_its_scenes(gpu, count):
    """The place bits shrink as the scenes grow in number; every image stays the scene's own."""
    packs = []
    for k in range(count):
        w = W.mid_scene(seed=k, rays_per_light=64 + k, n_objects=3 + k)
        w.params.width, w.params.height, w.params.max_bounce = 97 + k, 61, 6
        packs.append(w.packed())
    with Context() as ctx:
        images, _ = _batch(ctx, packs)
    with Context(culling=abi.LG_CULL_OFF) as ctx:
        for k in range(0, count, max(1, count // 7)):
            ctx.upload(packs[k])
            img, _ = ctx.render()
            assert np.array_equal(images[k], img), k
