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
