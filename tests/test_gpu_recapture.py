"""A frame rendered again after an edit that changes only how many rays a light has."""
import numpy as np
import pytest

from light_garden_gb300 import abi, workloads as W
from light_garden_gb300.runtime import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rays", [(4096, 1024), (1024, 4096), (512, 300_000)])
def test_ray_count_edit_renders_anew(gpu, rays):
    packs = [W.plain_small(accum=abi.LG_ACCUM_FIXED64, num_rays=n).packed() for n in rays]
    with Context() as ctx:
        for pk in packs:
            ctx.upload(pk)
            edited, st = ctx.render()
            assert st["ray_visits"] > pk.lights[0].num_rays
    with Context() as ctx:
        ctx.upload(packs[1])
        fresh, st2 = ctx.render()
    assert st["ray_visits"] == st2["ray_visits"] and np.array_equal(edited, fresh)
