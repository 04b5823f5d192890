"""The plan kernel (ports, window corners, residual shifts) against the FP64 oracle, bit for bit: no, some
and all radial coefficients, one to four sensors per thread, Bayer kernel offsets, and rounding at
ties, signs and the range where corners are clamped."""
import numpy as np
import pytest

from helpers import make_gpu, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,w,h,dist", [
    ("quad_mono", 128, 96, [0.0] * 7),
    ("quad_mono", 136, 40, [-0.1, 0.02] + [0.0] * 5),
    ("quad_bayer", 96, 72, [0.03, -0.02, 0.01, 0.0, 0.002, -0.001, 0.0005]),
    ("circle_lwir", 96, 80, [0.0, 0.0, 0.05] + [0.0] * 4),
    ("quad_bayer", 1296, 968, [0.0] * 7),  # more tasks than one per-sensor wave: four sensors a thread
])
def test_ports_and_corners_bit_exact(oracle, kind, w, h, dist):
    from tileproc import synth
    sc = synth.make_scene(kind, seed=81, width=w, height=h)
    g = sc["geometry"]
    g["distortion"] = dist
    S, C = g["num_sensors"], sc["num_colors"]
    rng = np.random.default_rng(17)
    for k, s in (("azimuth", 2e-3), ("tilt", 2e-3), ("roll", 5e-3), ("zoom", 5e-3)):
        g[k] = (s * rng.standard_normal(S)).tolist()
    g["azimuth"][0] = g["tilt"][0] = g["roll"][0] = g["zoom"][0] = 0.0
    T = (w // 8) * (h // 8)
    target = rng.uniform(-4, 8, T).astype(np.float32)
    target[::5] = 0.0
    k = e = None
    if C == 3:
        k, e = synth.random_clt_kernels(rng, S, h // 16 + 2, w // 16 + 2, C)
        e[0, ..., 0:8] = 0.0  # exact ties and zero offsets
    ref = run_oracle(oracle, sc, target, kernels=k, kext=e, corr=False)
    with make_gpu(sc, k, e) as tp:
        tp.setFullFrameImages(target)
        tp.execPorts()
        tl, res = tp.getSubtiles()
        assert np.array_equal(tp.getPorts(), ref["ports"])
    # both sides in task order (every tile)
    assert np.array_equal(tl.reshape(ref["int_tl"].shape), ref["int_tl"])
    assert np.array_equal(res.reshape(ref["residual"].shape), ref["residual"].astype(np.float32))


def _java_round(x):
    f = np.floor(x)
    return np.where(x - f >= 0.5, f + 1, f)


@pytest.mark.parametrize("step", [16, 12])
def test_corner_rounding_of_given_ports(step):
    """Ports given as tasks: ties of both signs, a hair beside them, zero, the clamped range; a kernel
    step that is no power of two."""
    from tileproc import GPUTileProcessor
    w, h, kv, kh = 64, 64, 8, 8
    x = np.array([8.0, 8.5, 7.5, 9.5, 6.5, 8.0 + 2.0 ** -20, np.nextafter(np.float32(8.5), np.float32(0)),
                  np.nextafter(np.float32(8.5), np.float32(9)), np.nextafter(np.float32(7.5), np.float32(0)), -3.5, -4.5,
                  0.0, -1e-30, 1e-30, 63.5, 64.0, w + 1024.0, w + 1023.5, -1024.0, -1023.5, 8.25, 20.0, 28.0, 36.0],
                 np.float32)
    n = len(x)
    xy = np.stack([x, x[::-1]], -1)[:, None].repeat(4, 1)
    rng = np.random.default_rng(2)
    ext = np.zeros((4, kv, kh, 1, 8), np.float32)
    ext[1:, ..., 0:2] = rng.uniform(-0.5, 0.5, (3, kv, kh, 1, 2))
    ext[1:, ..., 4:8] = rng.uniform(-0.01, 0.01, (3, kv, kh, 1, 4))
    kern = np.zeros((4, kv, kh, 1, 4, 64), np.float32)
    kern[..., 0, :] = 1
    with GPUTileProcessor(4, w, h, kernels_hor=kh, kernels_vert=kv, kernel_step=step) as tp:
        tp.setConvolutionKernels(kern, ext)
        tp.setBayerImages(np.zeros((4, h, w), np.float32))
        tp.setTasks(tp.packTasks(np.ones(n), np.arange(n) % 8, np.arange(n) // 8, xy))
        tp.execPorts()
        tl, res = tp.getSubtiles()
    c = xy.astype(np.float64)
    kt = np.clip(_java_round(c / step) + 1, 0, [kh - 1, kv - 1]).astype(int)
    kd = c - (kt - 1 + 0.5) * step
    e = ext[np.arange(4)[None], kt[..., 1], kt[..., 0], 0].astype(np.float64)
    off = np.stack([e[..., 0] + e[..., 4] * kd[..., 0] + e[..., 5] * kd[..., 1],
                    e[..., 1] + e[..., 6] * kd[..., 0] + e[..., 7] * kd[..., 1]], -1)
    p = (c - 8) - off
    t = -_java_round(-p)
    lo, hi = -(1024 + 16), 64 + 1024
    par = np.abs(t) % 2
    want = np.where(t > hi, hi - ((hi % 2) != par), np.where(t < lo, lo + ((lo % 2) != par), t))
    assert np.array_equal(tl[:, :, 0], want.astype(int))
    assert np.array_equal(res[:, :, 0], (-(p - t)).astype(np.float32))


@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 128 * 1024, 128 * 1024 + 1, 300001])
def test_compaction_sizes(n):
    """One block, block edges, the largest list whose blocks count for themselves and the first beyond."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    from tileproc import _lib as L
    lib = L.load()
    rng = np.random.default_rng(n)
    op = np.where(rng.random(n) < 0.3, rng.integers(1, 99, n), 0).astype(np.int32)
    op[-1] = 7
    d = rng.random(n).astype(np.float32)
    dop, dd = torch.from_numpy(op).cuda(), torch.from_numpy(d).cuda()
    out = torch.zeros((3, n), dtype=torch.int32, device="cuda")
    num = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert lib.tp_compact_tile_ops_noalloc(p(dop), p(dd), 640, n, p(out[0]), p(out[1]), p(out[2]), p(num), None) == L.TP_OK
    torch.cuda.synchronize()
    i = np.nonzero(op)[0]
    k = int(num.item())
    assert k == len(i)
    got = out[:, :k].cpu().numpy()
    assert np.array_equal(got[0], (i % 640) | ((i // 640) << 16))
    assert np.array_equal(got[1], op[i]) and np.array_equal(got[2].view(np.float32), d[i])


def test_tile_map_follows_the_task_list():
    """IMCLT reads the tile -> task map: sparse tile ops, then packed tasks, then tile ops again, against
    handles that saw only one list."""
    from tileproc import synth
    sc = synth.make_scene("quad_mono", seed=5, width=128, height=96)
    T = 16 * 12
    rng = np.random.default_rng(3)
    ops = [(rng.random(T) < f).astype(np.int32) for f in (0.5, 0.7)]
    i = np.nonzero(rng.random(T) < 0.4)[0]
    with make_gpu(sc) as tp:
        tp.setFullFrameImages(2.0)
        tp.execPorts()
        xy = tp.getPorts()[i].astype(np.float32)
        packed = tp.packTasks(np.ones(len(i)), i % 16, i // 16, xy)

    def frame(tp, step):
        if step == 1:
            tp.setTasks(packed)
        else:
            tp.setFullFrameImages(2.0, tile_op=ops[step // 2])
        tp.execConverCorrectTiles()
        tp.execImcltRbg()
        return tp.getRBG(1)
    with make_gpu(sc) as tp:
        got = [frame(tp, k) for k in range(3)]
    for k in range(3):
        with make_gpu(sc) as tp:
            assert np.array_equal(got[k], frame(tp, k))


def test_padded_and_packed_images():
    from tileproc import GPUTileProcessor, synth
    import ctypes as C
    from tileproc import _lib as L
    sc = synth.make_scene("quad_mono", seed=6, width=64, height=48)
    res = []
    for pad in (0, 24):
        with GPUTileProcessor(4, 64, 48) as tp:
            tp.setGeometry(sc["geometry"])
            for s in range(4):
                a = np.full((48, 64 + pad), np.nan, np.float32)
                a[:, :64] = sc["images"][s]
                tp._ck(tp._lib.tp_set_image(tp.h, s, C.c_void_p(a.ctypes.data), L.TP_F32, 64 + pad), "tp_set_image")
            tp.setCorrelation()
            tp.setFullFrameImages(3.0)
            tp.process()
            res.append((tp.getClt(), tp.getDisparity()))
    assert np.array_equal(res[0][0], res[1][0]) and np.array_equal(res[0][1], res[1][1], equal_nan=True)
