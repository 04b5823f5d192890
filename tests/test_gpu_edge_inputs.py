"""Forms and inputs at the edge of the standard quads' and many-pair kernels: strips of more than 32 entries of u16
Bayer quads and of batched mono quads, tiles without a peak in the many-pair adjoint, and pixels that are NaN or
infinite.  Each against the general kernels (another order of the pairs, one camera's image of the other type, the
warp-per-tile schedule) or the same scene alone, on the same inputs."""
import numpy as np
import pytest

from helpers import make_gpu
from test_gpu_quad import ORDER, PAIRS, _run, _scene
from tileproc import synth
from tileproc.batch import Batch

pytestmark = pytest.mark.gpu

LONG = {"corr_strip_hight": 5, "corr_wndy_size": 4}  # 60 strip entries


@pytest.mark.parametrize("w,h,fill,kw", [(16, 16, 1.0, LONG), (136, 72, 0.5, LONG), (72, 40, 1.0, {"corr_strip_hight": 16, "corr_wndy_size": 16})])
def test_long_strips_of_u16_bayer_quads(w, h, fill, kw):
    sc = _scene("quad_bayer", True, w, h, 71)
    T = (w // 8) * (h // 8)
    rng = np.random.default_rng(w)
    op = (rng.uniform(size=T) < fill).astype(np.int32)
    op[0] = op[-1] = 1
    target = rng.uniform(0, 8, T).astype(np.float32)
    kernels = synth.random_clt_kernels(rng, 4, h // 16 + 2, w // 16 + 2, 3)
    got = _run(sc, kernels, PAIRS, op, target, kw)
    want = _run(sc, kernels, PAIRS, op, target, kw, mixed=True)
    on = op != 0
    assert np.array_equal(got[0][on], want[0][on])
    assert np.array_equal(got[1][on], want[1][on], equal_nan=True)
    assert np.array_equal(got[2], want[2], equal_nan=True)


@pytest.mark.parametrize("u16", [False, True])
def test_long_strips_in_a_batch_of_mono_quads(u16):
    sizes = [(16, 16), (136, 72), (72, 40)]
    tps = [make_gpu(_scene("quad_mono", u16, w, h, 75 + i)) for i, (w, h) in enumerate(sizes)]
    try:
        for i, (tp, (w, h)) in enumerate(zip(tps, sizes)):
            tp.setCorrelation(**(LONG if i else {}))  # one scene with a short strip among them
            tp.setFullFrameImages(np.full((w // 8) * (h // 8), 3.0, np.float32))
            tp.process()
        want = [(tp.getCorr(), tp.getDisparity()) for tp in tps]
        with Batch(tps) as b:
            for _ in range(2):
                b.run_graph()
                b.synchronize()
                for tp, (c, d) in zip(tps, want):
                    assert np.array_equal(tp.getCorr(), c, equal_nan=True)
                    assert np.array_equal(tp.getDisparity(), d, equal_nan=True)
    finally:
        for tp in tps:
            tp.close()


@pytest.mark.parametrize("S,w,h,kern", [(5, 40, 24, False), (16, 96, 64, True)])
def test_many_pair_adjoint_with_tiles_without_a_peak(S, w, h, kern):
    rng = np.random.default_rng(S)
    g = synth.circle_geometry(S, w, h, rng=rng, sigma=2e-4)
    img = synth.lowpass_noise(rng, h + 16, w + 16)
    img = np.stack([img[8:8 + h, 8:8 + w]] * S) + 0.02 * rng.normal(size=(S, h, w))
    img = np.clip(np.rint(2048 + 400 * img), 0, 4095).astype(np.uint16)
    img[:, :, : w // 2] = 0  # windows of zeros: no correlation, no peak
    T = (w // 8) * (h // 8)
    kernels = synth.random_clt_kernels(rng, S, h // 16 + 2, w // 16 + 2, 1, strength=0.05) if kern else (None, None)
    sc = dict(geometry=g, num_colors=1, width=w, height=h, images=img)
    out = []
    for mixed in (False, True):
        with make_gpu(sc, *kernels) as tp:
            if mixed:  # the general kernel
                tp.setBayerImage(img[0].astype(np.float32), 0)
            tp.setCorrelation(pairs=synth.circle_pairs(g))
            tp.setFullFrameImages(0.0)
            tp.setAdjointMode(False)
            tp.process()
            tp.backward()
            out.append((tp.getPortSensitivities(), tp.getDisparityJacobian()[2]))
    (s0, d0), (s1, d1) = out
    none = np.isnan(d0)
    assert none.any() and not none.all() and np.array_equal(none, np.isnan(d1))
    assert (s0[none] == 0).all()
    # the same sums in another order, relative to the tile's largest sensitivity
    scale = np.abs(s1).reshape(T, -1).max(1)[:, None, None]
    assert np.all(np.abs(s0 - s1) <= 2e-5 * np.maximum(scale, 1e-6))


def _spoil(images, value):
    images[1, 10, 21] = value   # an inner pixel of one sensor, a corner pixel of another (read mirrored too)
    images[-1, 0, 0] = value


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("kind,w,h,kern", [("quad_mono", 72, 40, False), ("quad_bayer", 72, 40, True)])
def test_nan_and_infinite_pixels_in_quads(value, kind, w, h, kern):
    sc = _scene(kind, False, w, h, 77)
    _spoil(sc["images"], value)
    T = (w // 8) * (h // 8)
    rng = np.random.default_rng(6)
    target = rng.uniform(0, 4, T).astype(np.float32)
    op = np.ones(T, np.int32)
    kernels = synth.random_clt_kernels(rng, 4, h // 16 + 2, w // 16 + 2, sc["num_colors"]) if kern else None
    clt, corr, disp = _run(sc, kernels, PAIRS, op, target, {})
    gclt, gcorr, gdisp = _run(sc, kernels, [PAIRS[i] for i in ORDER], op, target, {})
    bad = ~np.isfinite(clt).all(axis=(2, 3, 4))
    assert bad[:, 1].any() and bad[:, 3].any() and not bad[:, [0, 2]].any() and not bad.all(1).any()
    assert np.array_equal(clt, gclt, equal_nan=True)
    assert np.array_equal(corr[:, ORDER], gcorr, equal_nan=True)
    hit = bad.any(1)
    assert np.array_equal(np.isfinite(disp), np.isfinite(gdisp))
    same = (disp[:, 8] == gdisp[:, 8]) | np.isnan(disp[:, 8])
    assert same[~hit].mean() > 0.9
    # the strip product takes the pairs in another order: a few ulp of the geometric mean
    np.testing.assert_allclose(disp[same], gdisp[same], rtol=2e-5, atol=2e-5, equal_nan=True)
    # a pair whose two sensors are sound keeps its surface: that of a scene without the pixel
    sc["images"][~np.isfinite(sc["images"])] = 0
    _, ccorr, cdisp = _run(sc, kernels, PAIRS, op, target, {})
    for i, p in enumerate(PAIRS):
        sound = ~(bad[:, p[0]] | bad[:, p[1]])
        assert np.array_equal(corr[sound, i], ccorr[sound, i], equal_nan=True)
    assert np.array_equal(disp[~hit], cdisp[~hit], equal_nan=True)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_nan_and_infinite_pixels_in_many_pairs(value):
    from tileproc import GPUTileProcessor
    S, w, h = 7, 72, 40
    rng = np.random.default_rng(8)
    g = synth.circle_geometry(S, w, h, rng=rng)
    pairs = [list(p) for p in synth.circle_pairs(g)]
    img = rng.normal(size=(h + 16, w + 16))
    img = (np.stack([img[s % 5:s % 5 + h, s % 7:s % 7 + w] for s in range(S)])
           + 0.05 * rng.normal(size=(S, h, w))).astype(np.float32)
    clean = img.copy()
    _spoil(img, value)
    T = (w // 8) * (h // 8)
    out = []
    for images, sched in ((img, (0, 0)), (img, (2, 2)), (clean, (0, 0))):
        with GPUTileProcessor(S, w, h) as tp:
            tp.setGeometry(g)
            tp.setBayerImages(images)
            tp.setCorrelation(pairs=pairs)
            tp.setSchedule(*sched)
            tp.setFullFrameImages(np.full(T, 2.0, np.float32))
            tp.process()
            out.append((tp.getClt(), tp.getCorr(), tp.getDisparity()))
    (clt, corr, d), (gclt, gcorr, gd), (_, ccorr, cd) = out
    bad = ~np.isfinite(clt).all(axis=(2, 3, 4))
    assert bad[:, 1].any() and bad[:, -1].any() and not bad[:, [0, 2, 3, 4, 5]].any()
    assert np.array_equal(clt, gclt, equal_nan=True) and np.array_equal(corr, gcorr, equal_nan=True)
    assert np.array_equal(np.isfinite(d), np.isfinite(gd))
    same = (d[:, 8] == gd[:, 8]) | np.isnan(d[:, 8])
    # the mean of 21 logarithms in another order
    np.testing.assert_allclose(d[same], gd[same], rtol=1e-4, atol=1e-4, equal_nan=True)
    for i, p in enumerate(pairs):
        sound = ~(bad[:, p[0]] | bad[:, p[1]])
        assert np.array_equal(corr[sound, i], ccorr[sound, i], equal_nan=True)
    assert np.array_equal(d[~bad.any(1)], cd[~bad.any(1)], equal_nan=True)


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("kind,kern", [("quad_mono", False), ("quad_bayer", True)])
def test_nan_and_infinite_pixels_in_the_conversion(value, kind, kern):
    """The conversion stage: the sub-tiles whose colour holds the pixel, and no others, are not finite, as in the fused
    forward; the others are those of a scene without it."""
    w, h = 72, 40
    sc = _scene(kind, False, w, h, 79)
    clean = sc["images"].copy()
    rng = np.random.default_rng(5)
    kernels = synth.random_clt_kernels(rng, 4, h // 16 + 2, w // 16 + 2, sc["num_colors"]) if kern else (None, None)
    out = []
    _spoil(sc["images"], value)
    for images in (sc["images"], clean):
        with make_gpu(dict(sc, images=images), *kernels) as tp:
            tp.setCorrelation()
            tp.setFullFrameImages(2.0)
            tp.execConverCorrectTiles()
            stage = tp.getClt()
            tp.process()
            out.append((stage, tp.getClt()))
    (stage, fused), (cstage, _) = out
    bad = ~np.isfinite(stage).all(axis=(3, 4))
    assert bad.any() and np.array_equal(bad, ~np.isfinite(fused).all(axis=(3, 4)))
    assert np.array_equal(stage[~bad], cstage[~bad])
