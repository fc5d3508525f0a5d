"""Reading an FP32 accumulation takes little device memory however large the image: it is rounded from
the FP64 sums in pieces."""
import numpy as np
import pytest

from light_garden_gb300 import abi, workloads as W

pytestmark = pytest.mark.gpu


def test_accum_download_takes_little_memory(ctx):
    import torch

    w = W.plain_small(accum=abi.LG_ACCUM_F32, num_rays=512)
    w.params.width, w.params.height = 4093, 3071
    pk = w.packed()
    ctx.upload(pk)
    first, _ = ctx.render()
    free = torch.cuda.mem_get_info()[0]
    acc = ctx.accum()
    assert torch.cuda.mem_get_info()[0] >= free - (40 << 20)  # the image is 201 MB
    again, _ = ctx.render()
    assert np.array_equal(first, again)
    assert np.array_equal(acc.astype(np.float16).view(np.uint16), first)  # the resolve rounds the same FP32 values
