"""Full raster units: enough (segment, tile) pairs that every unit holds the most segments its mode allows
(16384 in fixed point, 1024 in FP32), all on the same pixels, with terms whose split parts are the
largest there are, so that the 32-bit plane sums come next to 2^31 on either side.  The sum of a pixel is
the number of segments times the term."""
import numpy as np
import pytest

from light_garden_gb300 import abi
from test_gpu_raster import _image, _params

pytestmark = pytest.mark.gpu

N = 244_000       # segments across 128 tiles: 31.2 M pairs, more than three units of 16384 a raster CTA
ROW = 21          # the pixel row (column) that all are in


def _bundle(tall, colors):
    """N equal segments along the whole canvas; tall: down a 64 x 4096 canvas, else along 4096 x 64."""
    w, h = (64, 4096) if tall else (4096, 64)
    segs = np.zeros(N, abi.segment_dtype())
    end = 1.0 if tall else w / h
    side = ((ROW + 0.5) - w / 2) / (h / 2) if tall else 1.0 - (ROW + 0.5) / (h / 2)
    a, b = ("y", "x") if tall else ("x", "y")
    segs[a + "0"], segs[a + "1"], segs[b + "0"], segs[b + "1"] = -end, end, side, side
    segs["color"] = colors
    return w, h, segs


def _line(img, tall):
    line = img[:, ROW] if tall else img[ROW]
    rest = np.delete(img, ROW, axis=1 if tall else 0)
    return line, rest


@pytest.mark.parametrize("tall", [False, True])
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("terms", [
    (4 - 2.0 ** -22, 2 - 2.0 ** -23, 1 - 2.0 ** -24),          # the largest high parts
    ((2 ** 24 - 1) * 2.0 ** -32, 1 - 2.0 ** -24, 0.0),         # the largest low part; staged in two reads
])
def test_fixed_point(gpu, oracle, terms, sign, tall):
    w, h, segs = _bundle(tall, tuple(sign * t for t in terms) + (1.0,))
    p = _params(w, h, abi.LG_ACCUM_FIXED64)
    p.clear_color[:] = (0.0, 0.0, 0.0, 0.0)
    img, pixels = _image(p, segs)
    assert pixels == N * 4096
    line, rest = _line(img, tall)
    want = np.array([N * int(sign * t * 2 ** 32) for t in terms] + [N << 32], np.int64)  # whole numbers of 2^-32
    assert np.array_equal(line, np.broadcast_to(want, line.shape))
    assert not rest.any()


@pytest.mark.parametrize("tall", [False, True])
@pytest.mark.parametrize("sign", [1, -1])
def test_f32(gpu, oracle, sign, tall):
    # one brighter segment sets the unit; then the largest high part, the largest low part, and both
    terms = (1 - 2.0 ** -24, (2 ** 24 - 1) * 2.0 ** -42, 0.75)
    colors = np.tile(np.array([sign * t for t in terms] + [1.0], np.float32), (N, 1))
    colors[0, 1] = sign * 0.75
    w, h, segs = _bundle(tall, colors)
    p = _params(w, h, abi.LG_ACCUM_F32)
    p.clear_color[:] = (0.0, 0.0, 0.0, 0.0)
    img, pixels = _image(p, segs)
    assert pixels == N * 4096
    line, rest = _line(img, tall)
    want = np.array([sign * N * terms[0], sign * ((N - 1) * terms[1] + 0.75), sign * N * terms[2], float(N)])
    # a unit's sum is exact; an FP64 rounding for each of the 239 units and one to FP32
    tol = 2.0 ** -24 * np.abs(want) + 240 * 2.0 ** -52 * np.abs(want)
    assert (np.abs(line.astype(np.float64) - want) <= tol).all()
    assert not rest.any()
