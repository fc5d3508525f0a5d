"""A negative zero among a curved mirror's control points keeps its sign in the control lines."""
import numpy as np
import pytest

from light_garden_gb300 import abi
from light_garden_gb300.scene import CubicBezier, Object, pack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.LG_PRECISION_EXACT, abi.LG_PRECISION_FAST])
def test_control_lines_keep_signed_zeros(gpu, oracle, precision):
    from light_garden_gb300.runtime import Context

    params = abi.params_default()
    params.width, params.height, params.precision = 96, 64, precision
    mirrors = [CubicBezier(((-0.0, 0.0), (0.1, -0.0), (0.0, 0.3), (0.4, 0.3))),
               CubicBezier(((0.0, -0.0), (-0.0, -0.1), (-0.3, 0.0), (-0.0, -0.0)))]
    pk = pack([Object.new_curved_mirror(m) for m in mirrors], [], params)
    with Context() as ctx:
        ctx.upload(pk)
        ctx.trace()
        segs = ctx.segments()
    want = oracle.trace(pk)[0]
    assert len(want) == 6
    assert sorted(s.tobytes() for s in segs) == sorted(s.tobytes() for s in want)
