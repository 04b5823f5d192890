"""A packed task list may name a tile more than once.  Every forward that hands its strip and profile products to
a separate extraction pass then finishes the tile once per entry; with the same ports in every entry, the record
is that of a list without repeats, bit for bit.  The repeats lie at the other end of the list and next to their
tile; the forwards are the standard quads' (mono, float Bayer, u16 Bayer with short and long strips), u16 Bayer
quads with the pairs in another order, many general pairs, and a batch of mono quads."""
import numpy as np
import pytest

from helpers import make_gpu
from test_gpu_quad import ORDER, PAIRS
from tileproc import synth
from tileproc.batch import Batch

pytestmark = pytest.mark.gpu

W, H = 136, 72
NX, T = W // 8, (W // 8) * (H // 8)


def _handle(kind, u16, pairs, kw):
    if kind == "circle":
        sc = synth.make_scene("circle_lwir", seed=83, width=W, height=H)
        pairs = synth.circle_pairs(sc["geometry"])
    else:
        sc = synth.make_scene(kind, seed=83, width=W, height=H)
        if kind == "quad_bayer" and not u16:
            sc["images"] = sc["images"].astype(np.float32)
    tp = make_gpu(sc)
    tp.setCorrelation(pairs=pairs, **kw)
    tp.setFullFrameImages(np.random.default_rng(3).uniform(0, 6, T).astype(np.float32))
    tp.execPorts()
    return tp, tp.getPorts().astype(np.float32)


def _tasks(ports, tiles):
    from tileproc import GPUTileProcessor
    tiles = np.asarray(tiles)
    return GPUTileProcessor.packTasks(np.ones(len(tiles), np.int32), tiles % NX, tiles // NX, ports[tiles])


# 153 tiles: 100 of them, then again the first and the last of them and one in the middle, twice in a row
UNIQUE = np.arange(T - 100, T)
REPEAT = np.r_[UNIQUE[:50], UNIQUE[49], UNIQUE[50:], UNIQUE[0], UNIQUE[0], UNIQUE[-1], UNIQUE[:30]]


def _results(tp):
    return tp.getClt()[UNIQUE], tp.getCorr()[UNIQUE], tp.getDisparity()


@pytest.mark.parametrize("kind,u16,pairs,kw", [
    ("quad_mono", False, PAIRS, {}),
    ("quad_mono", False, PAIRS, {"corr_strip_hight": 5, "corr_wndy_size": 4}),
    ("quad_bayer", False, PAIRS, {}),
    ("quad_bayer", True, PAIRS, {}),
    ("quad_bayer", True, PAIRS, {"corr_strip_hight": 5, "corr_wndy_size": 4}),
    ("quad_bayer", True, [PAIRS[i] for i in ORDER], {}),
    ("circle", False, None, {}),
])
def test_repeated_tiles_give_the_record_of_one(kind, u16, pairs, kw):
    tp, ports = _handle(kind, u16, pairs, kw)
    with tp:
        tp.setTasks(_tasks(ports, UNIQUE))
        tp.process()
        want = _results(tp)
        assert np.isfinite(want[2][UNIQUE, 1]).mean() > 0.5
        for _ in range(3):
            tp.setTasks(_tasks(ports, REPEAT))
            tp.process()
            for a, b in zip(_results(tp), want):
                assert np.array_equal(a, b, equal_nan=True)


def test_repeated_tiles_in_a_batch():
    made = [_handle("quad_mono", False, PAIRS, {}) for _ in range(2)]
    tps = [m[0] for m in made]
    try:
        tp, ports = made[0]
        tp.setTasks(_tasks(ports, UNIQUE))
        tp.process()
        want = _results(tp)
        for tp, ports in made:
            tp.setTasks(_tasks(ports, REPEAT))
        with Batch(tps) as b:
            for step in (lambda: b.process(replan=True), b.run_graph):
                step()
                b.synchronize()
                for tp in tps:
                    for x, y in zip(_results(tp), want):
                        assert np.array_equal(x, y, equal_nan=True)
    finally:
        for tp in tps:
            tp.close()
