"""A small frame's generations in one launch each against three launches.

A frame of few rays and objects takes each generation through the search, the solve and the
bounce in one kernel; an explicit number of pair slots asks for the three kernels.  Both answer
with the same bits, path for path, on either side of the rule and where a ray has more candidates
than its list holds.
"""
import numpy as np
import pytest

from light_garden_gb300 import abi, workloads as W
from light_garden_gb300.runtime import Context
from light_garden_gb300.scene import Circle, Material, Object, PointLight, pack

pytestmark = pytest.mark.gpu


def _rings(n, rays):
    """Concentric discs about two lights: every ray is inside all of them."""
    objects = [Object(abi.LG_OBJ_CIRCLE, Circle((0.0, 0.0), 0.1 + 0.03 * k), Material(1.1 + 0.02 * k)) for k in range(n)]
    lights = [PointLight((0.01, 0.02), rays, (1.0, 0.5, 0.25, 1.0)), PointLight((-0.02, 0.0), rays, (0.2, 0.5, 1.0, 1.0))]
    params = abi.params_default()
    params.width, params.height, params.max_bounce = 333, 241, 6
    return pack(objects, lights, params)


def _scene(name):
    kind, n, rays = name.split("-")
    n, rays = int(n), int(rays)
    if kind == "rings":
        return _rings(n, rays)
    if kind == "csg":
        w = W.csg_scene(seed=n, total_rays=rays, n_objects=n, width=320, height=200, string_mod=False)
    elif kind == "mid":
        w = W.mid_scene(seed=n, rays_per_light=rays, n_objects=n)
    else:
        w = W.shapes_scene(seed=n, rays_per_light=rays, n_objects=n)
    w.params.width, w.params.height, w.params.max_bounce = 319, 203, 7
    return w.packed()


def _render(pk, **kw):
    with Context(**kw) as ctx:
        ctx.upload(pk)
        st = ctx.trace()
        segs, paths = ctx.segments(paths=True)
        ctx.accumulate()
        acc = ctx.accum()
        img, st2 = ctx.render()
    order = np.lexsort((paths["path"], paths["gen"], paths["primary"], paths["light"], paths["source"]))
    return st, segs[order], paths[order], acc, img, st2


@pytest.mark.parametrize("name", ["rings-1-1", "rings-7-31", "rings-9-33", "rings-24-65", "rings-25-65", "csg-1-257",
                                  "csg-8-4099", "csg-9-4099", "mid-24-2048", "mid-25-2048", "mid-3-8192",
                                  "mid-3-8193", "shapes-12-1023", "shapes-23-4097"])
@pytest.mark.parametrize("stride", [1, 3])
def test_one_launch_is_three_launches(gpu, name, stride):
    pk = _scene(name)
    pk.params.precision, pk.params.accum = abi.LG_PRECISION_EXACT, abi.LG_ACCUM_FIXED64
    pk.params.record_paths = 1
    pk.params.ray_stride, pk.params.ray_offset = stride, stride - 1
    a, b = _render(pk), _render(pk, scan_pairs=16)
    for k in ("ray_visits", "segments", "primary_rays"):
        assert a[0][k] == b[0][k], k
    assert a[1].tobytes() == b[1].tobytes()
    for f in ("source", "light", "primary", "gen", "path", "hit"):
        assert np.array_equal(a[2][f], b[2][f]), f
    keep = np.uint8(0xff & ~(abi.LG_PATH_FALLBACK | abi.LG_PATH_NEAR_DEGENERATE))  # routes and reported bands
    assert np.array_equal(a[2]["flags"] & keep, b[2]["flags"] & keep)
    assert np.array_equal(a[3], b[3]) and np.array_equal(a[4], b[4])
