"""Crossings of a string mod's lines (nested mods) against the oracle: the same points in the same
order, for counts around a warp, a row and a block of pairs, for lines that share end points
(decided in FP64), for curves that leave FP32's comfortable range, and without any crossing."""
import numpy as np
import pytest

from light_garden_gb300 import abi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("curve", [0, 1, 2, 3])
@pytest.mark.parametrize("m", [2, 3, 6, 17, 64, 65, 257, 600])
def test_nested_lines_match_oracle(gpu, oracle, curve, m):
    from light_garden_gb300.runtime import Context

    pk = W.nested_string_mod_art(curve=curve, width=128, height=96, outer_modulo=m).packed()
    with Context() as ctx:
        ctx.upload(pk)
        ctx.trace()
        got = ctx.chords()
    want = oracle.string_mod_chords(pk.params)
    assert len(got) == len(want)
    assert got.tobytes() == want.tobytes()


def test_growing_spiral_matches_oracle(gpu, oracle):
    """|c| > 1: the points span many orders of magnitude, up to where FP32 overflows."""
    from light_garden_gb300.runtime import Context

    pk = W.nested_string_mod_art(curve=abi.LG_CURVE_COMPLEX_EXP, width=64, height=64, outer_modulo=300).packed()
    pk.params.string_mod.curve_f[0], pk.params.string_mod.curve_f[1] = 1.2, 0.9
    with Context() as ctx:
        ctx.upload(pk)
        ctx.trace()
        got = ctx.chords()
    want = oracle.string_mod_chords(pk.params)
    assert got.tobytes() == want.tobytes()
