"""The kernels of standard quads (tp_quad.cu) against the general forward: the same pairs in another
order, or one camera of another image type, take the general path, whose surfaces are the same bits.
Sizes: a single row of tiles, widths whose staged windows end at the row's end, an odd tile count;
a strip of more than 32 entries; a sparse task list; a batch of the mono forms."""
import numpy as np
import pytest

from helpers import make_gpu

pytestmark = pytest.mark.gpu

PAIRS = [(0, 1, 0, 1, 1., 0.), (2, 3, 0, 1, 1., 0.), (0, 2, 1, 1, 0., 1.), (1, 3, 1, 1, 0., 1.),
         (0, 3, 2, 1, 1., 1.), (2, 1, 3, 1, 1., -1.)]
ORDER = [1, 0, 3, 2, 4, 5]


def _scene(kind, u16, w, h, seed):
    from tileproc import synth
    sc = synth.make_scene(kind, seed=seed, width=w, height=h)
    if kind == "quad_mono" and u16:
        sc["images"] = np.clip(np.rint(2048 + 400 * sc["images"]), 0, 4095).astype(np.uint16)
    if kind == "quad_bayer" and not u16:
        sc["images"] = sc["images"].astype(np.float32)
    return sc


def _run(sc, kernels, pairs, op, target, corr_kw, mixed=False):
    k, e = kernels if kernels else (None, None)
    with make_gpu(sc, k, e) as tp:
        if mixed:  # the same pixel values, one camera as float
            tp.setBayerImage(sc["images"][3].astype(np.float32), 3)
        tp.setCorrelation(pairs=pairs, **corr_kw)
        tp.setFullFrameImages(target, tile_op=op)
        tp.process()
        tp.process()
        return tp.getClt(), tp.getCorr(), tp.getDisparity()


@pytest.mark.parametrize("kind,u16,w,h,fill,kern,corr_kw", [
    ("quad_mono", False, 16, 16, 1.0, False, {}),
    ("quad_mono", False, 136, 72, 1.0, False, {}),
    ("quad_mono", True, 200, 24, 0.5, False, {}),
    ("quad_mono", True, 72, 136, 1.0, False, {"corr_strip_hight": 5, "corr_wndy_size": 4}),
    ("quad_bayer", True, 104, 88, 1.0, True, {}),
    ("quad_bayer", False, 88, 104, 0.6, True, {}),
    ("quad_bayer", False, 24, 200, 1.0, False, {"corr_wndy_size": 3}),
])
def test_quad_path_matches_general_path(kind, u16, w, h, fill, kern, corr_kw):
    from tileproc import synth
    sc = _scene(kind, u16, w, h, 61)
    T = (w // 8) * (h // 8)
    rng = np.random.default_rng(9)
    op = (rng.uniform(size=T) < fill).astype(np.int32)
    op[0] = op[-1] = 1
    target = rng.uniform(0, 8, T).astype(np.float32)
    kernels = synth.random_clt_kernels(rng, 4, h // 16 + 2, w // 16 + 2, sc["num_colors"]) if kern else None
    clt, corr, disp = _run(sc, kernels, PAIRS, op, target, corr_kw)
    gclt, gcorr, gdisp = _run(sc, kernels, [PAIRS[i] for i in ORDER], op, target, corr_kw)
    on = op != 0
    assert np.array_equal(clt[on], gclt[on])
    assert np.array_equal(corr[on][:, ORDER], gcorr[on], equal_nan=True)
    # the strip product takes the pairs in another order: a few ulp of the geometric mean
    assert np.array_equal(np.isnan(disp), np.isnan(gdisp))
    same_max = (disp[:, 8] == gdisp[:, 8]) | np.isnan(disp[:, 8])
    assert same_max.mean() > 0.99
    ok = on & same_max
    np.testing.assert_allclose(disp[ok], gdisp[ok], rtol=2e-5, atol=2e-5, equal_nan=True)
    if u16:
        mclt, mcorr, mdisp = _run(sc, kernels, PAIRS, op, target, corr_kw, mixed=True)
        assert np.array_equal(clt[on], mclt[on]) and np.array_equal(corr[on], mcorr[on], equal_nan=True)
        assert np.array_equal(disp, mdisp, equal_nan=True)


@pytest.mark.parametrize("u16", [False, True])
def test_quad_batch_matches_single_scenes(u16):
    from tileproc.batch import Batch
    sizes = [(16, 16), (136, 72), (72, 40)]
    scenes = [_scene("quad_mono", u16, w, h, 70 + i) for i, (w, h) in enumerate(sizes)]
    rng = np.random.default_rng(4)
    tps = [make_gpu(sc) for sc in scenes]
    try:
        for tp, (w, h) in zip(tps, sizes):
            T = (w // 8) * (h // 8)
            tp.setCorrelation()
            tp.setFullFrameImages(rng.uniform(0, 8, T).astype(np.float32),
                                  tile_op=np.r_[1, (rng.uniform(size=T - 1) < 0.8)].astype(np.int32))
            tp.process()
        want = [tp.getDisparity() for tp in tps]
        with Batch(tps) as b:
            for _ in range(2):
                b.run_graph()
                b.synchronize()
                for tp, d in zip(tps, want):
                    assert np.array_equal(tp.getDisparity(), d, equal_nan=True)
    finally:
        for tp in tps:
            tp.close()


@pytest.mark.parametrize("w,h,fill,combo,kw,kern", [
    (16, 16, 1.0, [1, 1, 1, 1, 1, 1], {}, True),                       # four tiles
    (24, 200, 1.0, [1, 0, 1, 1, 0, 1], {"twice_diagonal": 0}, False),  # odd and even tiles, pairs not combined
    (136, 72, 0.4, [0, 1, 1, 0, 1, 1], {}, True),                      # sparse
    (648, 24, 1.0, [1, 1, 1, 1, 1, 1], {"corr_wndy_size": 1}, True),   # strips of 15 entries
])
def test_three_warp_bayer_quads_match_general_path(w, h, fill, combo, kw, kern):
    """u16 Bayer quads with short strips (a warp per colour, then per couple of pairs) against the general path: the
    same pairs with one camera's image as float.  The order of operations is the same, so the results are the same
    bits, the strips' products included."""
    from tileproc import synth
    sc = _scene("quad_bayer", True, w, h, 67)
    T = (w // 8) * (h // 8)
    rng = np.random.default_rng(11)
    op = (rng.uniform(size=T) < fill).astype(np.int32)
    op[0] = op[-1] = 1
    target = rng.uniform(0, 8, T).astype(np.float32)
    kernels = synth.random_clt_kernels(rng, 4, h // 16 + 2, w // 16 + 2, 3) if kern else None
    pairs = [p[:3] + (c,) + p[4:] for p, c in zip(PAIRS, combo)]
    got = _run(sc, kernels, pairs, op, target, kw)
    want = _run(sc, kernels, pairs, op, target, kw, mixed=True)
    on = op != 0
    assert np.array_equal(got[0][on], want[0][on])
    assert np.array_equal(got[1][on], want[1][on], equal_nan=True)
    assert np.array_equal(got[2], want[2], equal_nan=True)
