"""The scan's launch shape by rule (lg_device_opts.scan_pairs = 0): the table with 16 pair slots a lane
below 48 objects, the grid walk with 8 from there on.  Either gives the bits of every fixed choice and
of the oracle."""
import numpy as np
import pytest

from light_garden_gb300 import abi, workloads as W
from parity import exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_objects", [15, 16, 47, 48])  # around the grid's and the walk's first size
def test_rule_and_fixed_shapes_agree(gpu, oracle, n_objects):
    from light_garden_gb300.runtime import Context

    w = W.mid_scene(seed=n_objects, accum=abi.LG_ACCUM_FIXED64, rays_per_light=1 << 12, n_objects=n_objects, n_lights=4)
    w.params.width, w.params.height, w.params.max_bounce, w.params.record_paths = 320, 180, 8, 1
    pk = w.packed()
    images = {}
    for pairs in (0, 8, 16):
        for culling in (abi.LG_CULL_AUTO, abi.LG_CULL_OFF, abi.LG_CULL_ON):
            with Context(scan_pairs=pairs, culling=culling) as ctx:
                ctx.upload(pk)
                ctx.trace()
                if pairs == 0 and culling == abi.LG_CULL_AUTO:
                    segs, paths = ctx.segments(paths=True)
                ctx.accumulate()
                images[pairs, culling] = ctx.accum()
    first = images[0, abi.LG_CULL_AUTO]
    for k, img in images.items():
        assert np.array_equal(img, first), k
    o_segs, o_paths, _, _ = oracle.trace(pk)
    rep = exact(segs, paths, o_segs, o_paths)
    assert rep.ok(), rep
