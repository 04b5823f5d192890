"""The render path (per-stage conversion, then IMCLT) at the sizes where its kernels can go wrong: regions of the
IMCLT that end at or one tile past the frame, both region sizes, windows that cross the image border, each colour
of a mosaic, u16 and float images, sparse task lists."""
import numpy as np
import pytest

from helpers import make_gpu
from tileproc import synth

pytestmark = pytest.mark.gpu


def _scene(kind, u16, w, h, seed):
    sc = synth.make_scene(kind, seed=seed, width=w, height=h)
    if kind == "quad_mono" and u16:
        sc["images"] = np.clip(np.rint(2048 + 400 * sc["images"]), 0, 4095).astype(np.uint16)
    if kind == "quad_bayer" and not u16:
        sc["images"] = sc["images"].astype(np.float32)
    return sc


@pytest.mark.parametrize("kind,w,h,fill", [
    ("quad_mono", 16, 16, 1.0),      # one region of 6x6 blocks, not filled
    ("quad_mono", 40, 88, 1.0),      # 6 and 12 blocks: regions that end with the frame
    ("quad_bayer", 48, 96, 0.5),     # one block past them
    ("quad_bayer", 392, 312, 1.0),   # 240 regions of 10x10 blocks, both sides end with the frame
    ("quad_bayer", 400, 320, 0.3),   # one block past them
])
def test_imclt_regions_match_oracle(oracle, kind, w, h, fill):
    """Max error 2e-6 of the largest value, as for the full frame: four FP32 products and sums of 8-point transforms."""
    sc = _scene(kind, True, w, h, 81)
    S, Cn, T = 4, sc["num_colors"], (w // 8) * (h // 8)
    rng = np.random.default_rng(5)
    op = (rng.uniform(size=T) < fill).astype(np.int32)
    op[0] = op[-1] = 1
    with make_gpu(sc) as tp:
        tp.setCorrelation()
        tp.setFullFrameImages(np.full(T, 3.0, np.float32), tile_op=op)
        tp.process()
        tp.execImcltRbg()
        clt = tp.getClt().astype(np.float64).reshape(T, S, Cn, 4, 64)
        got = [tp.getRBG(s).astype(np.float64) for s in range(S)]
    clt[op == 0] = 0
    want = oracle.imclt_frames(clt, w // 8, h // 8, scale=0.25, present=op)
    for s in range(S):
        assert np.abs(got[s].reshape(want[s].shape) - want[s]).max() < 2e-6 * np.abs(want[s]).max()


@pytest.mark.parametrize("kind,u16,w,h,fill,kern", [
    ("quad_bayer", True, 16, 16, 1.0, True),
    ("quad_bayer", True, 136, 72, 0.6, True),
    ("quad_bayer", False, 72, 104, 1.0, False),
    ("quad_mono", True, 72, 40, 1.0, False),
    ("quad_mono", False, 40, 72, 1.0, True),
])
def test_stage_conversion_matches_fused_forward(kind, u16, w, h, fill, kern):
    """The CLT of the conversion stage against the fused forward's (other transforms, the same values).  The fused one
    takes four factors from __sincosf (within 2^-21.4 each, 1.5e-6 together); the rest, 1e-6 of the largest
    coefficient, is for both sides' FP32 roundings, doubled."""
    sc = _scene(kind, u16, w, h, 82)
    T = (w // 8) * (h // 8)
    rng = np.random.default_rng(6)
    op = (rng.uniform(size=T) < fill).astype(np.int32)
    op[0] = op[-1] = 1
    target = rng.uniform(0, 12, T).astype(np.float32)
    k, e = synth.random_clt_kernels(rng, 4, h // 16 + 2, w // 16 + 2, sc["num_colors"]) if kern else (None, None)
    clts = []
    for staged in (False, True):
        with make_gpu(sc, k, e) as tp:
            tp.setCorrelation()
            tp.setFullFrameImages(target, tile_op=op)
            if staged:
                tp.execPorts()
                tp.execConverCorrectTiles()
            else:
                tp.process()
            clts.append(tp.getClt()[op != 0])
    assert np.abs(clts[0]).max() > 0
    assert np.abs(clts[1] - clts[0]).max() < 4e-6 * np.abs(clts[0]).max()
