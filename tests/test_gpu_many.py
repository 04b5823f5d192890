"""The kernel of mono scenes with many general pairs (tp_many.cu) against the warp-per-tile schedule: CLT
and surfaces bit for bit, the strips' combination (summed by another number of warps) to a few ulp.
Sensor counts that fill one to four groups, odd pair counts (a last pair alone), pairs left out of the
combination, both image types, kernel tables, sparse tasks."""
import numpy as np
import pytest

from tileproc import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,w,h,u16,kern,fill,drop", [
    (5, 16, 16, False, False, 1.0, 0),
    (6, 72, 40, False, True, 1.0, 0),    # 15 pairs
    (7, 40, 72, True, False, 0.5, 3),    # 21 pairs, 3 not combined
    (11, 88, 24, True, True, 1.0, 0),
    (16, 136, 88, False, False, 1.0, 1),
])
def test_many_pairs_match_warp_per_tile(S, w, h, u16, kern, fill, drop):
    from tileproc import GPUTileProcessor
    rng = np.random.default_rng(S)
    g = synth.circle_geometry(S, w, h, rng=rng)
    pairs = [list(p) for p in synth.circle_pairs(g)]
    for p in pairs[:drop]:
        p[3] = 0
    img = rng.normal(size=(h + 16, w + 16))
    img = np.stack([img[s % 5:s % 5 + h, s % 7:s % 7 + w] for s in range(S)]) + 0.05 * rng.normal(size=(S, h, w))
    img = np.clip(np.rint(2048 + 400 * img), 0, 4095).astype(np.uint16) if u16 else img.astype(np.float32)
    T = (w // 8) * (h // 8)
    op = (rng.uniform(size=T) < fill).astype(np.int32)
    op[0] = op[-1] = 1
    kh, kv = (w // 16 + 2, h // 16 + 2) if kern else (0, 0)
    out = []
    for sched in ((0, 0), (2, 2)):
        with GPUTileProcessor(S, w, h, kernels_hor=kh, kernels_vert=kv) as tp:
            tp.setGeometry(g)
            if kern:
                k, e = synth.random_clt_kernels(np.random.default_rng(1), S, kv, kh, 1)
                tp.setConvolutionKernels(k, e)
            tp.setBayerImages(img)
            tp.setCorrelation(pairs=pairs)
            tp.setSchedule(*sched)
            tp.setFullFrameImages(np.full(T, 2.0, np.float32), tile_op=op)
            tp.process()
            tp.process()
            out.append((tp.getClt(), tp.getCorr(), tp.getDisparity()))
    (clt, corr, d), (gclt, gcorr, gd) = out
    on = op != 0
    assert np.array_equal(clt[on], gclt[on]) and np.array_equal(corr[on], gcorr[on], equal_nan=True)
    assert np.array_equal(np.isnan(d), np.isnan(gd))
    same = (d[:, 8] == gd[:, 8]) | np.isnan(d[:, 8])
    assert same.mean() > 0.99
    # the mean of up to 120 logarithms in another order: 120 roundings at most
    np.testing.assert_allclose(d[same], gd[same], rtol=1e-4, atol=1e-4, equal_nan=True)
