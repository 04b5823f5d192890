"""A backward pass gives the same bits whatever the handle ran before: the first one, whose forward has not recorded
its strip samples, a repeated one, the one after a recording forward, and the first of a handle that records from the
start.  Many general pairs (tp_adjoint_many.cu) and Bayer quads (tp_adjoint_quad.cu), strips of one and two rows, pairs
left out, sparse tasks, both image types.  And all of them agree with the general kernel, which takes the same pixels
where one camera's image is of the other type."""
import numpy as np
import pytest

from helpers import make_gpu
from test_gpu_quad import PAIRS
from tileproc import synth

pytestmark = pytest.mark.gpu


def _scene(S, w, h, u16, rng):
    if S == 4:
        sc = synth.make_scene("quad_bayer", seed=37, width=w, height=h)
        pairs, op0 = [list(p) for p in PAIRS], sc["disparity_gt"].reshape(-1).astype(np.float32)
    else:
        g = synth.circle_geometry(S, w, h, rng=rng, sigma=3e-4)
        img = synth.lowpass_noise(rng, h + 16, w + 16)
        img = np.stack([img[8:8 + h, 8:8 + w]] * S) + 0.02 * rng.normal(size=(S, h, w))
        sc = dict(geometry=g, num_colors=1, width=w, height=h,
                  images=np.clip(np.rint(2048 + 400 * img), 0, 4095).astype(np.uint16))
        pairs, op0 = [list(p) for p in synth.circle_pairs(g)], np.zeros((w // 8) * (h // 8), np.float32)
    if not u16:
        sc["images"] = sc["images"].astype(np.float32)
    return sc, pairs, op0


@pytest.mark.parametrize("S,w,h,u16,kern,fill,drop,kw", [
    (5, 16, 16, True, False, 1.0, (), {}),
    (9, 40, 72, False, True, 0.5, (3, 7), {}),
    (16, 96, 64, False, False, 1.0, (), {"corr_wndy_size": 1}),
    (4, 16, 16, True, False, 1.0, (), {}),
    (4, 72, 56, True, True, 0.6, (2, 5), {}),
    (4, 104, 40, False, True, 1.0, (0,), {"corr_wndy_size": 1}),
])
def test_first_backward_is_the_later_one(S, w, h, u16, kern, fill, drop, kw):
    rng = np.random.default_rng(40 + S)
    sc, pairs, target = _scene(S, w, h, u16, rng)
    for i in drop:
        pairs[i][3] = 0
    T = (w // 8) * (h // 8)
    op = (rng.uniform(size=T) < fill).astype(np.int32)
    op[0] = op[-1] = 1
    dl = rng.uniform(-1, 1, T).astype(np.float32)
    kernels = (synth.random_clt_kernels(rng, S, h // 16 + 2, w // 16 + 2, sc["num_colors"], strength=0.05)
               if kern else (None, None))

    def handle():
        tp = make_gpu(sc, *kernels)
        tp.setCorrelation(pairs=pairs, **kw)
        tp.setFullFrameImages(target, tile_op=op)
        return tp

    def back(tp):
        ge, gd = tp.backward(dl)
        return (ge, gd[op != 0], tp.getPortSensitivities()[op != 0]) + tuple(x[op != 0] for x in tp.getDisparityJacobian())

    got = []
    with handle() as tp:
        tp.process()
        got += [back(tp), back(tp)]
        tp.process()
        got.append(back(tp))
    with handle() as tp:
        tp.setAdjointMode(False)
        tp.process()
        got.append(back(tp))
    with handle() as tp:
        last = sc["images"][S - 1]
        tp.setBayerImage(last.astype(np.float32 if u16 else np.uint16), S - 1)
        tp.process()
        want = back(tp)
    assert np.isfinite(got[0][5]).any()
    for g in got[1:]:
        for a, b in zip(got[0], g):
            assert np.array_equal(a, b, equal_nan=True)
    # the general kernel: the same sums in another order, relative to the tile's largest sensitivity
    s0, s1 = want[2], got[0][2]
    scale = np.abs(s0).reshape(len(s0), -1).max(1)[:, None, None]
    assert np.all(np.abs(s0 - s1) <= 2e-5 * np.maximum(scale, 1e-6))
