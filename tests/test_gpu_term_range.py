"""FP32 sums over terms of very different sizes: the split sums' unit follows the largest term of each
channel, smaller terms are drawn in windows of 19 exponents below it, and what lies outside all windows
goes straight into the image."""
import numpy as np
import pytest

from light_garden_gb300 import abi
from test_gpu_raster import _image, _params, _segments

pytestmark = pytest.mark.gpu


def _colors(kind, n, rng):
    c = rng.uniform(0.25, 1.0, (n, 4))
    c[:, 3] = 1.0
    if kind == "faint alpha":      # its square, a channel of terms near 2^-19 beside colours near 1
        c[:, 3] = 0.75 * 2.0 ** -9
    elif kind == "saturated":      # terms on both sides of the first window's edge in one channel
        c *= 2.0 ** rng.integers(-10, 1, (n, 1))
        c[:, 1] *= 2.0 ** -9
        c[:, 2] = 0.0
        c[:, 3] = 1.0
    elif kind == "bright":
        c[:, :3] *= 2.0 ** rng.integers(-20, 12, (n, 1))
    elif kind == "edges":          # exponents at the windows' edges, mantissas all ones and all zeros
        e = rng.choice([0, -18, -19, -20, -37, -38, -39, -56, -57, -58, -100], (n, 3))
        c[:, :3] = np.where(rng.random((n, 3)) < 0.5, 1.0, 2.0 - 2.0 ** -23) * 2.0 ** e.astype(float) * rng.choice([-1, 1], (n, 3))
    elif kind == "wide":           # every FP32 exponent, denormals and zeros among them
        c[:, :3] *= 2.0 ** rng.integers(-149, 127, (n, 3)).astype(float)
        c[rng.random((n, 4)) < 0.1] = 0.0
    return c.astype(np.float32)


@pytest.mark.parametrize("op", [abi.LG_BO_ADD, abi.LG_BO_REVERSE_SUBTRACT])
@pytest.mark.parametrize("px", [4, 300])  # columns spread over the lanes, a lane per column
@pytest.mark.parametrize("kind", ["unit", "faint alpha", "saturated", "bright", "edges", "wide"])
def test_f32_sums_round_once(gpu, oracle, kind, px, op):
    for w, h, n in ((33, 65, 1), (257, 31, 260), (640, 480, 6000)):
        p = _params(w, h, abi.LG_ACCUM_F32)
        p.color_blend.op = op
        segs = _segments(n, w, h, px, "unit", n + px)
        segs["color"] = _colors(kind, n, np.random.default_rng(n))
        got, pixels = _image(p, segs)
        want, want_px = oracle.raster_f64(segs, p)
        mag, pa = segs.copy(), _params(w, h, abi.LG_ACCUM_F32)
        mag["color"] = np.abs(mag["color"])
        total, _ = oracle.raster_f64(mag, pa)
        assert pixels == want_px, (w, h, n)
        # half an FP32 ulp of the sum, and an FP64 rounding of the magnitudes for every term
        tol = 2.0 ** -24 * np.abs(want) + (n + 4) * 2.0 ** -52 * total + 2.0 ** -149
        with np.errstate(over="ignore"):
            big = np.abs(want) > np.finfo(np.float32).max
        assert np.array_equal(big, np.isinf(got))
        assert (np.abs(got.astype(np.float64) - want)[~big] <= tol[~big]).all(), (w, h, n)


def test_f32_without_allocation(gpu, oracle):
    """The caller's image has FP32 values: a rounding of the running sum for every unit and window."""
    import ctypes as C

    import torch

    w, h, n = 320, 200, 6000
    p = _params(w, h, abi.LG_ACCUM_F32)
    segs = _segments(n, w, h, 40, "unit", 3)
    segs["color"] = _colors("saturated", n, np.random.default_rng(4))
    dev = torch.from_numpy(segs.view(np.float32).reshape(-1, 8).copy()).cuda()
    img = torch.empty((h, w, 4), dtype=torch.float32, device="cuda")
    st = gpu.lg_accumulate_segments_noalloc(C.c_void_p(dev.data_ptr()), n, C.byref(p), C.c_void_p(img.data_ptr()),
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream), None)
    assert st == abi.LG_OK
    got = img.cpu().numpy().astype(np.float64)
    want, _ = oracle.raster_f64(segs, p)
    # a tile's refs in units of 256 and more, two orientations, three windows, at most
    adds = 2 * 3 * (n // 256 + 1)
    assert (np.abs(got - want) <= (adds + 1) * 2.0 ** -24 * want + 2.0 ** -149).all()  # no term is negative
