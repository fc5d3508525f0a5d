"""A growth of the device buffers that fails leaves no scene, not launches that go by capacities which
the buffers do not have.  The request is for more memory than any device has, so that the allocation
fails at once and takes nothing."""
import ctypes as C

import numpy as np
import pytest

from light_garden_gb300 import abi, workloads as W

pytestmark = pytest.mark.gpu


def test_growth_beyond_the_device_leaves_no_scene(gpu, ctx):
    pk = W.plain_small(accum=abi.LG_ACCUM_FIXED64, num_rays=512).packed()
    ctx.upload(pk)
    want, _ = ctx.render()
    one = np.zeros(1, abi.segment_dtype())
    st = gpu.lg_accumulate_segments(ctx.h, one.ctypes.data_as(C.POINTER(abi.lg_segment)), 1 << 40, None)
    assert st == abi.LG_ERR_OUT_OF_MEMORY
    for call in (ctx.render, ctx.trace, ctx.accumulate, ctx.segments, ctx.accum, ctx.resolve_f16, ctx.resolve_rgba8):
        with pytest.raises(abi.LgError) as e:
            call()
        assert e.value.status == abi.LG_ERR_NO_SCENE, call
    ctx.upload(pk)  # the capacities are first guesses again
    got, _ = ctx.render()
    assert np.array_equal(got, want)
    assert len(ctx.segments()) > 512
    # a batch takes the context as well
    ctx.batch_upload([pk])
    assert np.array_equal(ctx.batch_render()[0][0], want)
