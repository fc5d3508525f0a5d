"""The tile raster's paths at the sizes where they part: short segments (their columns spread
densely over a warp's lanes) and long ones (a lane per column), batches of one, a warp, a
round of the CTA and one more, tiles cut into many units, canvases that end inside a tile, and
terms outside the split sums' range (large, tiny, negative, zero, NaN)."""
import numpy as np
import pytest

from light_garden_gb300 import abi

pytestmark = pytest.mark.gpu

CANVASES = [(32, 32), (33, 65), (257, 31), (640, 480)]
COUNTS = [1, 33, 257, 6000]


def _segments(n, w, h, px, colors, seed):
    rng = np.random.default_rng(seed)
    segs = np.zeros(n, abi.segment_dtype())
    x, y = rng.uniform(-w / h, w / h, n), rng.uniform(-1, 1, n)
    a = rng.uniform(0, 2 * np.pi, n)
    length = rng.uniform(0.2, 1.0, n) * 2.0 * px / h
    segs["x0"], segs["y0"] = x, y
    segs["x1"], segs["y1"] = x + length * np.cos(a), y + length * np.sin(a)
    c = rng.uniform(0.0, 1.0, (n, 4)).astype(np.float32)
    c[:, 3] = 1.0
    if colors == "wide":
        k = rng.integers(0, 7, n)
        c[k == 1, :3] *= 9.0                      # above the split's range
        c[k == 2, :3] *= np.float32(-3.0)
        c[k == 3, 1] = np.float32(3e-7)           # below 2^-18, and below the fixed-point unit's half
        c[k == 4, 2] = np.float32(1e-12)
        c[k == 5, 0] = 0.0
        c[k == 6, 3] = 0.5
    segs["color"] = c
    return segs


def _params(w, h, accum):
    p = abi.params_default()
    p.width, p.height, p.accum = w, h, accum
    return p


def _image(p, segs):
    from light_garden_gb300.runtime import Context
    from light_garden_gb300.scene import pack

    with Context() as ctx:
        ctx.upload(pack([], [], p))
        st = ctx.accumulate_segments(segs)
        return ctx.accum(), st["pixels"]


@pytest.mark.parametrize("colors", ["unit", "wide"])
@pytest.mark.parametrize("px", [4, 300])
def test_fixed_point_bit_exact(gpu, oracle, px, colors):
    for ci, (w, h) in enumerate(CANVASES):
        for n in COUNTS:
            p = _params(w, h, abi.LG_ACCUM_FIXED64)
            segs = _segments(n, w, h, px, colors, 100 * ci + n)
            got, pixels = _image(p, segs)
            want, want_px = oracle.raster(segs, p)
            assert pixels == want_px, (w, h, n)
            assert np.array_equal(got, want), (w, h, n)


@pytest.mark.parametrize("colors", ["unit", "wide"])
@pytest.mark.parametrize("px", [4, 300])
def test_f32_sums_round_once(gpu, oracle, px, colors):
    """The F32 image is the FP64 sum of the terms rounded once: half an FP32 ulp of the sum, and
    n FP64 roundings of the terms' magnitudes (alpha is 1 or 1/2, so its square is exact)."""
    for ci, (w, h) in enumerate(CANVASES):
        for n in COUNTS:
            p = _params(w, h, abi.LG_ACCUM_F32)
            segs = _segments(n, w, h, px, colors, 100 * ci + n)
            got, pixels = _image(p, segs)
            want, want_px = oracle.raster_f64(segs, p)
            mag = segs.copy()
            mag["color"] = np.abs(mag["color"])
            total, _ = oracle.raster_f64(mag, p)
            assert pixels == want_px, (w, h, n)
            tol = 2.0 ** -24 * np.abs(want) + (n + 4) * 2.0 ** -52 * total + 2.0 ** -149
            assert (np.abs(got.astype(np.float64) - want) <= tol).all(), (w, h, n)


def test_nan_and_infinite_colours(gpu, oracle):
    """Fixed point adds nothing for NaN and clamps infinities; F32 carries both into the image."""
    w, h = 64, 48
    segs = _segments(40, w, h, 30, "unit", 5)
    segs["color"][3, 0] = np.nan
    segs["color"][7, 1] = np.inf
    p = _params(w, h, abi.LG_ACCUM_FIXED64)
    assert np.array_equal(_image(p, segs)[0], oracle.raster(segs, p)[0])
    p = _params(w, h, abi.LG_ACCUM_F32)
    got, want = _image(p, segs)[0], oracle.raster_f64(segs, p)[0]
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))


def test_f32_min_max(gpu):
    """Min and max keep the terms' own bits: the F32 image equals the fixed-point one's pattern."""
    w, h = 257, 131
    segs = _segments(3000, w, h, 60, "unit", 9)
    imgs = []
    for accum in (abi.LG_ACCUM_F32, abi.LG_ACCUM_FIXED64):
        p = _params(w, h, accum)
        p.color_blend = abi.lg_blend_component(abi.LG_BF_ONE, abi.LG_BF_ONE, abi.LG_BO_MAX)
        p.alpha_blend = abi.lg_blend_component(abi.LG_BF_ONE, abi.LG_BF_ONE, abi.LG_BO_MIN)
        imgs.append(_image(p, segs)[0])
    assert np.array_equal(np.rint(imgs[0].astype(np.float64) * 2.0 ** 32).astype(np.int64), imgs[1])
