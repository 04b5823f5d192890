"""The many-pair adjoint kernel (tp_adjoint_many.cu) against the general one: a handle's first backward
pass has no recorded strip samples and takes the general kernel, later ones the many-pair kernel.
Sensor counts that leave rounds, warps' second pairs and groups partly empty; short baselines (several
strip entries in a cell); pairs left out; both image types; kernel tables; sparse tasks."""
import numpy as np
import pytest

from tileproc import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,w,h,u16,kern,fill,drop,shrink", [
    (5, 16, 16, False, False, 1.0, 0, 1.0),
    (7, 72, 40, True, True, 1.0, 4, 1.0),
    (9, 40, 72, False, False, 0.5, 0, 0.3),
    (13, 64, 48, False, True, 1.0, 1, 1.0),
    (16, 96, 64, False, False, 1.0, 0, 1.0),
])
def test_many_pair_adjoint_matches_general(S, w, h, u16, kern, fill, drop, shrink):
    from tileproc import GPUTileProcessor
    rng = np.random.default_rng(100 + S)
    g = synth.circle_geometry(S, w, h, rng=rng, sigma=3e-4)
    g["rXY"] = (np.asarray(g["rXY"]) * shrink).tolist()
    pairs = [list(p) for p in synth.circle_pairs(g)]
    for p in pairs[:drop]:
        p[3] = 0
    img = synth.lowpass_noise(rng, h + 16, w + 16)
    img = np.stack([img[8:8 + h, 8:8 + w]] * S) + 0.02 * rng.normal(size=(S, h, w))
    img = np.clip(np.rint(2048 + 400 * img), 0, 4095).astype(np.uint16) if u16 else img.astype(np.float32)
    T = (w // 8) * (h // 8)
    op = (rng.uniform(size=T) < fill).astype(np.int32)
    op[0] = op[-1] = 1
    kh, kv = (w // 16 + 2, h // 16 + 2) if kern else (0, 0)
    dl = rng.uniform(-1, 1, T).astype(np.float32)
    with GPUTileProcessor(S, w, h, kernels_hor=kh, kernels_vert=kv) as tp:
        tp.setGeometry(g)
        if kern:
            tp.setConvolutionKernels(*synth.random_clt_kernels(rng, S, kv, kh, 1, strength=0.05))
        tp.setBayerImages(img)
        tp.setCorrelation(pairs=pairs)
        tp.setFullFrameImages(0.0, tile_op=op)
        got = []
        for _ in range(3):
            tp.process()
            ge, gd = tp.backward(dl)
            got.append((ge, gd, tp.getPortSensitivities()[op != 0], tp.getDisparityJacobian()))
    a, b, c = got
    on = op != 0
    d0, d1 = a[3][2][on], b[3][2][on]
    assert np.array_equal(np.isnan(d0), np.isnan(d1)) and np.isfinite(d0).any()
    np.testing.assert_array_equal(d0, d1)
    # Sums of up to S - 1 pairs' terms per CLT entry in another order, then sums of 2048 products per
    # sensitivity: FP32 rounding of the largest terms, relative to the tile's largest sensitivity
    s0, s1 = a[2], b[2]
    scale = np.abs(s0).reshape(len(s0), -1).max(1)[:, None, None]
    assert np.all(np.abs(s0 - s1) <= 2e-5 * np.maximum(scale, 1e-6))
    for x, y in zip(b[:3], c[:3]):  # and it repeats exactly
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("dark,w,h,u16,kern,fill,drop,flat,corr_kw", [
    (True, 72, 56, True, True, 1.0, (), False, {}),
    (False, 16, 16, True, False, 1.0, (), False, {}),
    (False, 72, 56, True, True, 1.0, (), True, {}),
    (False, 56, 72, False, True, 0.5, (0,), False, {}),
    (False, 104, 40, True, True, 1.0, (2, 5), False, {"corr_wndy_size": 1}),
    (False, 40, 40, False, False, 1.0, (1, 0), True, {}),
])
def test_bayer_quad_adjoint_matches_general(dark, w, h, u16, kern, fill, drop, flat, corr_kw):
    """The Bayer quad kernel (tp_adjoint_quad.cu) the same way: pairs and whole couples left out of the
    combination, a one-row strip, tiles without a peak, both image types, sparse tasks."""
    from helpers import make_gpu
    from test_gpu_quad import PAIRS
    sc = synth.make_scene("quad_bayer", seed=91, width=w, height=h)
    if flat:
        sc["images"][:, :, : w // 2] = 2048
    if dark:  # windows of zeros: no correlation, no peak
        sc["images"][:, :, : w // 2] = 0
    if not u16:
        sc["images"] = sc["images"].astype(np.float32)
    rng = np.random.default_rng(w)
    for k in ("azimuth", "tilt", "roll", "zoom"):
        sc["geometry"][k] = (2e-4 * rng.standard_normal(4)).tolist()
    pairs = [list(p) for p in PAIRS]
    for i in drop:
        pairs[i][3] = 0
    T = (w // 8) * (h // 8)
    op = (rng.uniform(size=T) < fill).astype(np.int32)
    op[0] = op[-1] = 1
    kernels = synth.random_clt_kernels(rng, 4, h // 16 + 2, w // 16 + 2, 3, strength=0.05) if kern else (None, None)
    got = []
    with make_gpu(sc, *kernels) as tp:
        tp.setCorrelation(pairs=pairs, **corr_kw)
        tp.setFullFrameImages(sc["disparity_gt"].reshape(-1).astype(np.float32), tile_op=op)
        for _ in range(3):
            tp.process()
            tp.backward()
            got.append((tp.getPortSensitivities()[op != 0], tp.getDisparityJacobian()[2][op != 0]))
    (s0, d0), (s1, d1), (s2, d2) = got
    np.testing.assert_array_equal(d0, d1)
    assert np.isfinite(d0).any()
    if dark:
        assert np.isnan(d0).any()
    # the same sums in another order, as above
    scale = np.abs(s0).reshape(len(s0), -1).max(1)[:, None, None]
    assert np.all(np.abs(s0 - s1) <= 2e-5 * np.maximum(scale, 1e-6))
    np.testing.assert_array_equal(s1, s2)
    np.testing.assert_array_equal(d1, d2)
