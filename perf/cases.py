"""The measured work of the tile processor: what a user's program has it do, through GPUTileProcessor,
Batch and the C ABI that they bind (include/tp.h).

A case is one call pattern ("use") on one camera:

  depth    images resident, new target disparities and tile ops, forward, disparity record read back
           (the disparity scan: the same frame measured again at other disparities)
  frame    a new frame from host memory: images up, tile ops, forward, IMCLT, disparity and colour
           frames read back
  render   the reference's GPU flow: packed tasks, convert and correct, IMCLT, colour frames read back
  texture  forward, RGBA texture tiles with their weights, tiles and aux records read back
  lma      forward and the LMA ("POLY") disparity pass
  adjoint  forward and adjoint: loss gradient and the disparity Jacobian
  batch    many small scenes as one captured batch step, every disparity record read back

Cameras: "quad" (4 sensors, the 6 quad pairs; 1 or 3 colours) and "circle" (mono sensors on a circle,
every pair).  Scenes are rendered from the seed on the GPU: band-limited texture with rectangles (1/f
for the thermal circle), a disparity surface with steps, sensor noise; 12-bit Bayer mosaics or floats.

Large results go to page-locked buffers that the program keeps, as a frame loop does; small calls use
the plain getters.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "imagej-elphel_gb300"))


# ---------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------
def _case(use, camera, width, height, sensors=4, colors=1, u16=False, kernels=False, fill=1.0, scenes=1, name=None):
    c = {"use": use, "camera": camera, "width": width, "height": height, "sensors": sensors, "colors": colors,
         "u16": u16, "kernels": kernels, "fill": fill, "scenes": scenes}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest whole frame: 192 tiles, every call waits for its result (interactive use, tests)
        _case("frame", "quad", 128, 96, name="frame_mono_128x96"),
        # one step of a disparity scan on a small mono quad
        _case("depth", "quad", 512, 384, name="depth_mono_512x384"),
        # one step of a disparity scan on the 5 Mpix Bayer quad with its aberration kernels: the largest
        _case("depth", "quad", 2592, 1936, colors=3, u16=True, kernels=True, name="depth_bayer_2592x1936"),
        # a later scan step: a third of the tiles left, float mosaics (flat-fielded), odd tile counts
        _case("depth", "quad", 1304, 984, colors=3, kernels=True, fill=0.35, name="depth_bayer_f32_1304x984"),
        # thermal camera, 16 sensors, all 120 pairs
        _case("depth", "circle", 640, 512, sensors=16, name="depth_lwir16_640x512"),
        # one iteration of the extrinsic calibration of that camera: forward and adjoint
        _case("adjoint", "circle", 640, 512, sensors=16, name="adjoint_lwir16_640x512"),
        # the same on a Bayer quad with kernels
        _case("adjoint", "quad", 648, 488, colors=3, u16=True, kernels=True, name="adjoint_bayer_648x488"),
        # the reference's default disparity: forward, then the LMA fits
        _case("lma", "quad", 648, 488, colors=3, u16=True, name="lma_bayer_648x488"),
        # the camera loop: a 1.2 Mpix Bayer quad frame up, disparity and corrected colour frames down
        _case("frame", "quad", 1296, 968, colors=3, u16=True, kernels=True, name="frame_bayer_1296x968"),
        # the call sequence of GPUTileProcessor.java: tasks, convert and correct, IMCLT
        _case("render", "quad", 640, 480, colors=3, kernels=True, name="render_bayer_640x480"),
        # texture tiles of a scene for its 3D model
        _case("texture", "quad", 640, 480, colors=3, u16=True, kernels=True, name="texture_bayer_640x480"),
        # many small scenes at once (a server): 16 mono quads as one graph
        _case("batch", "quad", 512, 384, scenes=16, name="batch_mono_16x512x384"),
    ]


def _side(rng, lo, hi):
    return 8 * max(lo // 8, min(hi // 8, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 8))))


def draw(rng):
    use = rng.choice(["depth", "depth", "depth", "frame", "render", "texture", "lma", "adjoint", "adjoint", "batch"])
    fill = rng.choice([1.0, 1.0, round(rng.uniform(0.05, 0.95), 2)])
    if use in ("depth", "adjoint") and rng.random() < 0.4:
        s = rng.randint(5, 16)
        return _case(use, "circle", _side(rng, 64, 640), _side(rng, 64, 512), sensors=s,
                     fill=1.0 if use == "adjoint" else fill)
    if use == "batch":
        return _case(use, "quad", _side(rng, 64, 512), _side(rng, 64, 384), scenes=rng.randint(2, 24))
    wmax, hmax = {"depth": (2592, 1936), "frame": (1296, 968), "render": (1296, 968), "texture": (768, 576),
                  "lma": (648, 488), "adjoint": (968, 728)}[use]
    colors = 3 if use in ("texture", "render") else rng.choice([1, 3])
    return _case(use, "quad", _side(rng, 64, wmax), _side(rng, 64, hmax), colors=colors, u16=rng.random() < 0.6,
                 kernels=colors == 3 and rng.random() < 0.6, fill=1.0 if use in ("adjoint", "lma", "texture") else fill)


# Work counted from the algorithm: 8-point fast DTTs (about 44 operations), per (tile, sensor, colour)
# fold + four 2D DTTs + kernel convolution + phase rotation, per pair the normalised products of each
# colour + four 2D DTTs + unfold.
_FL_CLT, _FL_PAIR, _FL_PAIR_C, _FL_IMCLT, _FL_TEX = 7600, 4000, 3840, 5500, 150000


def work(case):
    W, H, S, C = case["width"], case["height"], case["sensors"], case["colors"]
    T = (W // 8) * (H // 8)
    n = max(1, int(round(T * case["fill"])))
    P = 6 if case["camera"] == "quad" else S * (S - 1) // 2
    use, N = case["use"], case["scenes"]
    images = S * W * H * (2 if case["u16"] else 4)
    kern = S * C * (W // 16 + 2) * (H // 16 + 2) * (1024 + 32) if case["kernels"] else 0
    rbg = S * C * (W + 8) * (H + 8) * 4
    fl_clt, fl_pairs = n * S * C * _FL_CLT, n * P * (_FL_PAIR + C * _FL_PAIR_C)
    by, fl = images + kern + T * 8, fl_clt
    if use != "render":
        by, fl = by + T * 36, fl + fl_pairs
    if use in ("frame", "render"):
        by, fl = by + rbg, fl + n * S * C * _FL_IMCLT
    if use == "texture":
        by, fl = by + T * (12 * 1024 + 64), fl + n * (S * C * _FL_IMCLT + _FL_TEX)
    if use == "lma":  # a pair's surface sampled and fitted, a few iterations of five small fits
        by, fl = by + T * 16, fl + n * 60000
    if use == "adjoint":
        by, fl = by + T * S * 16 + T * 12 + S * 16, fl + 2 * (fl_clt + fl_pairs)
    return {"bytes": by * N, "flops": fl * N}


# ---------------------------------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------------------------------
_BAYER_ROW, _BAYER_COL = 0, 1  # red pixel; colours are R, B, G


def _geometry(case, gen):
    W, H, S = case["width"], case["height"], case["sensors"]
    if case["camera"] == "quad":
        rxy, focal, pixel = [[-0.5, -0.5], [0.5, -0.5], [-0.5, 0.5], [0.5, 0.5]], 4.5, 2.2
    else:
        a = [2 * math.pi * i / S for i in range(S)]
        rxy, focal, pixel = [[math.cos(t) / math.sqrt(2), math.sin(t) / math.sqrt(2)] for t in a], 4.9, 12.0
    # rotations of a few pixels at most, whatever the focal length
    e = (torch.randn((4, S), generator=gen, device="cuda", dtype=torch.float64) * (0.4 * 0.001 * pixel / focal)).tolist()
    return {"num_sensors": S, "width": W, "height": H, "focal_length": focal, "pixel_size": pixel,
            "distortion_radius": 2.8512, "distortion": [0.0] * 7, "rXY": rxy, "pXY0": [[W / 2.0, H / 2.0]] * S,
            "azimuth": e[0], "tilt": e[1], "roll": e[2], "zoom": e[3]}


def _pairs(case, geom):
    """(cam1, cam2, kind, in combination, direction x, y)"""
    r = geom["rXY"]
    if case["camera"] == "quad":
        return [(0, 1, 0, 1, 1., 0.), (2, 3, 0, 1, 1., 0.), (0, 2, 1, 1, 0., 1.), (1, 3, 1, 1, 0., 1.),
                (0, 3, 2, 1, 1., 1.), (2, 1, 3, 1, 1., -1.)]
    return [(a, b, 4, 1, r[b][0] - r[a][0], r[b][1] - r[a][1]) for a in range(len(r)) for b in range(a + 1, len(r))]


def _rotations(az, tl, rl, zm):
    """Rotation (with zoom) of each sensor from tensors of any shape: [..., 3, 3]"""
    ca, sa, ct, st = torch.cos(az), torch.sin(az), torch.cos(tl), torch.sin(tl)
    cr, sr = torch.cos(rl) * (1 + zm), torch.sin(rl) * (1 + zm)
    z, o = torch.zeros_like(ca), torch.ones_like(ca)

    def mat(*v):
        return torch.stack(v, -1).reshape(ca.shape + (3, 3))
    return mat(cr, sr, z, -sr, cr, z, z, z, o) @ (mat(o, z, z, z, ct, st, z, -st, ct) @ mat(ca, z, -sa, z, o, z, sa, z, ca))


def _port(geom, rot, rxy, qx, qy, d):
    """Pixel of a sensor (rotation rot, offset rxy) that sees centre-image point (qx, qy) at disparity d."""
    f = geom["focal_length"] / (0.001 * geom["pixel_size"])
    vx, vy = qx - 0.5 * geom["width"] - d * rxy[0], qy - 0.5 * geom["height"] - d * rxy[1]
    x, y, z = (rot[..., i, 0] * vx + rot[..., i, 1] * vy + rot[..., i, 2] * f for i in range(3))
    return x * f / z + 0.5 * geom["width"], y * f / z + 0.5 * geom["height"]


def _texture(gen, h, w, thermal, sigma=1.5):
    n = torch.fft.rfft2(torch.randn((h, w), generator=gen, device="cuda"))
    f2 = torch.fft.fftfreq(h, device="cuda")[:, None] ** 2 + torch.fft.rfftfreq(w, device="cuda")[None] ** 2
    f2[0, 0] = 1
    n = n / f2.sqrt() if thermal else n * torch.exp(-2 * (math.pi * sigma) ** 2 * f2)
    n[0, 0] = 0
    t = torch.fft.irfft2(n, s=(h, w))
    return t / t.std()


def _scene(case, seed):
    """Everything the inputs are made of, on the GPU."""
    W, H, S, C = case["width"], case["height"], case["sensors"], case["colors"]
    tx, ty, M = W // 8, H // 8, 32
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)

    def rand(*s):
        return torch.rand(s, generator=gen, device="cuda")

    geom = _geometry(case, gen)
    # disparity: a smooth surface from a coarse grid plus a few nearer rectangles
    dmax = 8.0 if case["camera"] == "quad" else 4.0
    d = torch.nn.functional.interpolate(rand(1, 1, 4, 5) * 0.5 * dmax, size=(ty, tx), mode="bicubic", align_corners=True)[0, 0]
    box = rand(6, 4).tolist()
    for a, b, c, e in box:
        y0, x0 = int(a * ty * 0.8), int(b * tx * 0.8)
        d[y0:y0 + max(1, int(0.3 * ty * e)), x0:x0 + max(1, int(0.3 * tx * c))] += 0.35 * dmax * e
    d = d.clamp(0, dmax).contiguous()
    thermal = case["camera"] == "circle"
    base = _texture(gen, H + 2 * M, W + 2 * M, thermal)
    k = max(4, (W * H) // 2500)
    r = rand(k, 5).cpu()
    for i in range(min(k, 400)):
        x0, y0, w, h = int(r[i, 0] * (W + 40)), int(r[i, 1] * (H + 40)), 3 + int(r[i, 2] * 21), 3 + int(r[i, 3] * 21)
        base[y0:y0 + h, x0:x0 + w] += 0.5 if r[i, 4] < 0.5 else -0.5
    planes = [base] if C == 1 else [base + 0.3 * _texture(gen, H + 2 * M, W + 2 * M, False, 3.0) for _ in range(2)] + [base]
    ys, xs = torch.meshgrid(torch.arange(H, device="cuda", dtype=torch.float32),
                            torch.arange(W, device="cuda", dtype=torch.float32), indexing="ij")
    f64 = {q: torch.tensor(geom[q], device="cuda", dtype=torch.float32) for q in ("azimuth", "tilt", "roll", "zoom")}
    rots = _rotations(f64["azimuth"], f64["tilt"], f64["roll"], f64["zoom"])
    xo, yo = torch.arange(W, device="cuda") % 2 == _BAYER_COL, torch.arange(H, device="cuda") % 2 == _BAYER_ROW
    images = []
    for s in range(S):
        qx, qy = xs.clone(), ys.clone()
        for _ in range(3):  # the point of the centre image that this pixel sees
            dd = d[(qy / 8).long().clamp(0, ty - 1), (qx / 8).long().clamp(0, tx - 1)]
            px, py = _port(geom, rots[s], geom["rXY"][s], qx, qy, dd)
            qx, qy = qx + (xs - px), qy + (ys - py)
        grid = torch.stack([(qx + M) * 2 / (W + 2 * M - 1) - 1, (qy + M) * 2 / (H + 2 * M - 1) - 1], -1)[None]
        v = [torch.nn.functional.grid_sample(p[None, None], grid, mode="bicubic", padding_mode="reflection",
                                             align_corners=True)[0, 0] for p in planes]
        if C == 3:
            red, blue = yo[:, None] & xo[None], ~yo[:, None] & ~xo[None]
            v = torch.where(red, v[0], torch.where(blue, v[1], v[2]))
        else:
            v = v[0]
        v = v + (0.02 if thermal else 0.01) * torch.randn((H, W), generator=gen, device="cuda")
        if case["u16"]:
            v = (2048 + 400 * v).round().clamp(0, 4095)
        elif C == 3:
            v = 2048 + 400 * v
        images.append(v.float())
    T = tx * ty
    target = (d + (2 * rand(ty, tx) - 1) * (0.0 if case["use"] == "adjoint" else 1.0)).reshape(-1).float()
    op = torch.zeros(T, dtype=torch.int32, device="cuda")
    n = max(1, int(round(T * case["fill"])))
    op[torch.argsort(rand(T))[:n]] = 0xF
    kern = ext = None
    if case["kernels"]:
        kv, kh = H // 16 + 2, W // 16 + 2
        kern = 0.1 * torch.randn((S, kv, kh, C, 4, 64), generator=gen, device="cuda")
        kern[..., 0, :] += 1.0
        ext = torch.zeros((S, kv, kh, C, 8), device="cuda")
        ext[..., 0:2] = rand(S, kv, kh, C, 2) - 0.5
        ext[..., 2:4] = ext[..., 0:2]
        ext[..., 4:8] = 0.02 * rand(S, kv, kh, C, 4) - 0.01
    lpf = torch.exp(-0.02 * (torch.arange(8.)[:, None] ** 2 + torch.arange(8.)[None] ** 2)).reshape(1, 64).repeat(C, 1)
    return {"geometry": geom, "images": torch.stack(images), "target": target, "op": op, "kernels": kern, "ext": ext,
            "lpf": lpf, "pairs": _pairs(case, geom), "scales": [1.0, 1.0, 0.5]}


# ---------------------------------------------------------------------------------------------------
# the program's side
# ---------------------------------------------------------------------------------------------------
def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True)


def _address(t):
    return ctypes.c_void_p(t.data_ptr())


class _Camera:
    """A handle with its set-up, and the host buffers its program keeps."""

    def __init__(self, case, seed):
        from tileproc import GPUTileProcessor
        from tileproc import _lib as L
        sc = _scene(case, seed)
        W, H, S, C = case["width"], case["height"], case["sensors"], case["colors"]
        kh, kv = (W // 16 + 2, H // 16 + 2) if case["kernels"] else (0, 0)
        torch.cuda.synchronize()
        self.case = case
        self.images = sc["images"].cpu()
        if case["u16"]:  # the bits of the 12-bit samples
            self.images = self.images.to(torch.int16)
        self.images = self.images.pin_memory()
        self.frames = [a.numpy().view(np.uint16) if case["u16"] else a.numpy() for a in self.images]
        self.dtype = L.TP_U16 if case["u16"] else L.TP_F32
        self.target, self.op = sc["target"].cpu().numpy(), sc["op"].cpu().numpy()
        self.tp = tp = GPUTileProcessor(S, W, H, num_colors=C, kernels_hor=kh, kernels_vert=kv,
                                        bayer_red_row=_BAYER_ROW, bayer_red_col=_BAYER_COL)
        tp.setGeometry(sc["geometry"])
        if case["kernels"]:
            tp.setConvolutionKernels(sc["kernels"].cpu().numpy(), sc["ext"].cpu().numpy(), layout=L.TP_KERNELS_CPU)
        if C == 3:
            tp.setColorScales(sc["scales"])
        if case["use"] != "frame":
            tp.setBayerImages(self.frames)
        if case["use"] in ("frame", "render"):
            tp.setLpfRbg(sc["lpf"].numpy())
        if case["use"] != "render":
            tp.setCorrelation(pairs=None if case["camera"] == "quad" else sc["pairs"])
        T = tp.tilesX * tp.tilesY
        self.tiles = T
        self.disp = _pinned(T, 9)
        if case["use"] in ("frame", "render"):
            self.rbg = [_pinned(C, H + 8, W + 8) for _ in range(S)]
        if case["use"] == "texture":
            tp.setTextureParams()
            self.tex, self.aux = _pinned(T, 12, 256), _pinned(T, 16)
        if case["use"] == "render":  # packed tasks, as a Java host hands them over
            i = np.nonzero(self.op)[0]
            ports = _ports(sc, case, torch.tensor(i, device="cuda"))[0].float().cpu().numpy()
            self.tasks = tp.packTasks(np.full(len(i), 0xF), i % tp.tilesX, i // tp.tilesX, ports)

    def call(self, name, *args):
        self.tp._ck(getattr(self.tp._lib, name)(self.tp.h, *args), name)

    def disparity(self):
        """The disparity record into the program's buffer, in stream order."""
        self.call("tp_get_disparity_async", _address(self.disp), None)
        return self.disp


def prepare(case, seed):
    if case["use"] != "batch":
        return _Camera(case, seed)
    from tileproc.batch import Batch
    cams = [_Camera(case, seed * 64 + i) for i in range(case["scenes"])]
    for c in cams:
        c.tp.setFullFrameImages(c.target, tile_op=c.op)
    return {"cams": cams, "batch": Batch([c.tp for c in cams])}


def run(state):
    if isinstance(state, dict):
        state["batch"].run_graph()
        return [c.disparity() for c in state["cams"]]
    cam, tp = state, state.tp
    use, small = cam.case["use"], cam.tiles <= 1024
    if use == "render":
        tp.setTasks(cam.tasks)
        tp.execConverCorrectTiles()
        tp.execImcltRbg()
        for s in range(tp.num_sensors):
            cam.call("tp_get_rbg_async", s, _address(cam.rbg[s]), None)
        return cam.rbg
    if use == "frame":
        for s in range(tp.num_sensors):
            if small:
                tp.setBayerImage(cam.frames[s], s)
            else:
                cam.call("tp_set_image_async", s, _address(cam.images[s]), cam.dtype, 0, None)
    tp.setFullFrameImages(cam.target, tile_op=cam.op)
    tp.process()
    if use == "depth":
        return tp.getDisparity() if small else cam.disparity()
    if use == "frame":
        tp.execImcltRbg()
        if small:
            return [tp.getDisparity()] + [tp.getRBG(s) for s in range(tp.num_sensors)]
        for s in range(tp.num_sensors):
            cam.call("tp_get_rbg_async", s, _address(cam.rbg[s]), None)
        return [cam.disparity()] + cam.rbg
    if use == "texture":
        tp.execTextures()
        cam.call("tp_get_textures", _address(cam.tex))
        cam.call("tp_get_texture_aux", _address(cam.aux))
        return {"tex": cam.tex, "aux": cam.aux, "disparity": cam.disparity()}
    if use == "lma":
        return {"lma": tp.lmaRefine(), "disparity": cam.disparity()}
    ge, gd = tp.backward()
    je, jd, d = tp.getDisparityJacobian()
    return {"grad_extrinsics": ge, "grad_disparity": gd, "jac_extrinsics": je, "jac_disparity": jd, "disparity": d}


# ---------------------------------------------------------------------------------------------------
# the same in 64 bits, from the definitions
# ---------------------------------------------------------------------------------------------------
_F = torch.float64


def _t(x, **kw):
    return torch.tensor(x, dtype=_F, device="cuda", **kw)


def _dtt_tables():
    k, n = np.arange(8)[:, None], np.arange(8)[None]
    dct4 = 0.5 * np.cos(np.pi / 8 * (k + 0.5) * (n + 0.5))
    dst4 = 0.5 * np.sin(np.pi / 8 * (k + 0.5) * (n + 0.5))
    c2e = 0.5 * np.cos(np.pi * k * (2 * n + 1) / 16)
    s2e = ((-1.0) ** n) * c2e[7 - np.arange(8)]
    # fold of 16 samples to 8 for the cosine (0) and sine (1) branch, with the sine window and its quadrature
    w = np.sin(np.pi / 16 * (np.arange(8) + 0.5))
    fold = np.zeros((2, 2, 8, 16))  # branch, (cos, sin) of the shift, row, sample
    for x in range(8):
        if x < 4:
            terms = [(11 - x, 4 + x, 3 - x, -1, 1, -1), (12 + x, 3 - x, 4 + x, -1, -1, -1)]
        else:
            i = x - 4
            terms = [(i, i, 7 - i, 1, 1, 1), (7 - i, 7 - i, i, -1, 1, 1)]
        for src, win, dwin, sc, ss, ds in terms:
            for b, sg in ((0, sc), (1, ss)):
                fold[b, 0, x, src] += sg * w[win]
                fold[b, 1, x, src] += sg * w[dwin] * ds
    unfold = np.zeros((2, 16, 8))
    for j in range(16):
        seg, x = j >> 2, j & 3
        i = (x + 4, 7 - x, 3 - x, x)[seg]
        win = w[j if j < 8 else 15 - j]
        unfold[0, j, i] = win if seg == 0 else -win
        unfold[1, j, i] = -win if seg == 3 else win
    inv = [dct4, dst4]
    return {"fwd": _t(np.stack([[inv[b] @ fold[b, p] for p in range(2)] for b in range(2)])),
            "inv": _t(np.stack([unfold[b] @ inv[b] for b in range(2)])), "c2": _t(np.stack([c2e, s2e]))}


def _ports(sc, case, tiles, extr=None, disp=None):
    """Ports [n][S] x, y of the tiles (64 bits); extr [n][S][4] and disp [n] override the scene's (for derivatives)."""
    g, tx = sc["geometry"], case["width"] // 8
    if extr is None:
        extr = torch.stack([_t(g[k]) for k in ("azimuth", "tilt", "roll", "zoom")], -1)[None]
    if disp is None:
        disp = sc["target"][tiles].to(_F)
    rot = _rotations(*extr.unbind(-1))
    r = _t(g["rXY"])
    cx, cy = ((tiles % tx) * 8 + 4).to(_F)[:, None], ((tiles // tx) * 8 + 4).to(_F)[:, None]
    x, y = _port(g, rot, (r[:, 0], r[:, 1]), cx, cy, disp[:, None])
    return torch.stack([x, y], -1), disp


def _clt(sc, case, tab, ports):
    """CLT [n][S][C][4][8 (horizontal)][8 (vertical)] of windows at the ports [n][S][2]."""
    W, H, S, C = case["width"], case["height"], case["sensors"], case["colors"]
    n = ports.shape[0]
    dev = ports.device
    out = []
    sidx = torch.arange(S, device=dev)[None].expand(n, S)
    for c in range(C):
        p = ports - 8
        if sc["kernels"] is not None:
            kv, kh = sc["kernels"].shape[1:3]
            kt = torch.floor(ports.detach() / 16 + 0.5).long() + 1
            ktx, kty = kt[..., 0].clamp(0, kh - 1), kt[..., 1].clamp(0, kv - 1)
            e = sc["ext"][sidx, kty, ktx, c].to(_F)
            kd = ports - (torch.stack([ktx, kty], -1) - 1 + 0.5) * 16
            p = p - torch.stack([e[..., 0] + e[..., 4] * kd[..., 0] + e[..., 5] * kd[..., 1],
                                 e[..., 1] + e[..., 6] * kd[..., 0] + e[..., 7] * kd[..., 1]], -1)
        tl = -torch.floor(-p.detach() + 0.5)
        res = tl - p
        k16 = torch.arange(16, device=dev)
        col, row = tl[..., 0].long()[..., None] + k16, tl[..., 1].long()[..., None] + k16
        par_x, par_y = col % 2, row % 2
        col = torch.where(col < 0, par_x, torch.where(col >= W, W - 2 + par_x, col))
        row = torch.where(row < 0, par_y, torch.where(row >= H, H - 2 + par_y, row))
        win = sc["images"][sidx[..., None, None], row[..., :, None], col[..., None, :]].to(_F)
        if C == 3:
            ry, rx = (par_y == _BAYER_ROW)[..., :, None], (par_x == _BAYER_COL)[..., None, :]
            keep = (ry & rx, ~ry & ~rx, ry ^ rx)[c]
            win = win * keep * sc["scales"][c]
        a = math.pi / 16 * res
        w = torch.stack([torch.cos(a), torch.sin(a)], -1)  # [n][S][xy][2]
        mh = torch.einsum("nsp,bpfx->nsbfx", w[..., 0, :], tab["fwd"])
        mv = torch.einsum("nsp,bpfy->nsbfy", w[..., 1, :], tab["fwd"])
        q = torch.einsum("nsgvy,nsyx,nsbhx->nsgbhv", mv, win, mh)  # vertical branch g, horizontal branch b
        o = [q[:, :, 0, 0], q[:, :, 0, 1], q[:, :, 1, 0], q[:, :, 1, 1]]
        if sc["kernels"] is not None:
            k = sc["kernels"][sidx, kty, ktx, c].to(_F).reshape(n, S, 4, 8, 8).unbind(2)
            o = [o[0] * k[0] - o[1] * k[1] - o[2] * k[2] + o[3] * k[3], o[1] * k[0] + o[0] * k[1] - o[3] * k[2] - o[2] * k[3],
                 o[2] * k[0] - o[3] * k[1] + o[0] * k[2] - o[1] * k[3], o[3] * k[0] + o[2] * k[1] + o[1] * k[2] + o[0] * k[3]]
        f = (2 * torch.arange(8, device=dev) + 1).to(_F)
        ch, sh = torch.cos(a[..., 0, None] * f)[..., :, None], torch.sin(a[..., 0, None] * f)[..., :, None]
        cv, sv = torch.cos(a[..., 1, None] * f)[..., None, :], torch.sin(a[..., 1, None] * f)[..., None, :]
        t = [o[0] * ch - o[1] * sh, o[1] * ch + o[0] * sh, o[2] * ch - o[3] * sh, o[3] * ch + o[2] * sh]
        out.append(torch.stack([t[0] * cv - t[2] * sv, t[1] * cv - t[3] * sv, t[2] * cv + t[0] * sv, t[3] * cv + t[1] * sv], 2))
    return torch.stack(out, 2)


_FAT_ZERO, _SIGMA, _OFFSET, _MIN_CORR = (float(np.float32(v)) for v in (0.05, 0.8, 0.1, 0.02))  # the defaults
_RED, _BLUE = 0.5, float(np.float32(0.2))


def _corr_lpf(tab):
    i = np.arange(8)
    fd = np.exp(-(i[:, None] ** 2 + i[None] ** 2) / (2 * _SIGMA))
    c = np.cos(np.pi * i / 16) * np.where(i > 0, 2.0, 1.0)
    fd /= (fd * c[:, None] * c[None]).sum()
    k = np.arange(8)
    e = np.where((k == 0) | (k == 7), 0.5, 1.0)
    c3 = 0.5 * e[None] * np.cos(k[None] * (2 * k[:, None] + 1) * np.pi / 16)
    return _t(16 * c3 @ fd @ c3.T)  # [h][v] (symmetric)


def _corr(clt, tab, lpf, pairs):
    """Correlation surfaces [n][P][15][15] of the pairs."""
    i1, i2 = [p[0] for p in pairs], [p[1] for p in pairs]
    C = clt.shape[2]
    g = 1.0 / (1.0 + _RED + _BLUE)
    wt = [1.0] if C == 1 else [_RED * g, _BLUE * g, g]
    acc = 0
    for c in range(C):
        a, b = clt[:, i1, c].unbind(2), clt[:, i2, c].unbind(2)  # four [n][P][8][8]
        m = torch.sqrt(sum(x * x for x in a) * sum(x * x for x in b))
        m = m + m.mean((-1, -2), keepdim=True) * _FAT_ZERO ** 2
        t = [a[0] * b[0] + a[1] * b[1] + a[2] * b[2] + a[3] * b[3], -a[1] * b[0] + a[0] * b[1] - a[3] * b[2] + a[2] * b[3],
             -a[2] * b[0] - a[3] * b[1] + a[0] * b[2] + a[1] * b[3], a[3] * b[0] - a[2] * b[1] - a[1] * b[2] + a[0] * b[3]]
        acc = acc + torch.stack(t, 2) * (wt[c] / m)[:, :, None]
    acc = acc * lpf
    u = torch.stack([torch.einsum("yv,nphv,xh->npyx", tab["c2"][q >> 1], acc[:, :, q], tab["c2"][q & 1]) for q in range(4)])
    pad = torch.nn.functional.pad
    A, B, Cc, D = u[0], pad(u[1][..., :7], (1, 0)), pad(u[2][..., :7, :], (0, 0, 1, 0)), pad(u[3][..., :7, :7], (1, 0, 1, 0))
    f = lambda x, d: torch.flip(x, d)  # noqa: E731
    br, bl, tr, tl = A + B + Cc + D, A - B + Cc - D, A + B - Cc - D, A - B - Cc + D
    top = torch.cat([f(tl[..., 1:, 1:], (-1, -2)), f(tr[..., 1:, :], (-2,))], -1)
    bot = torch.cat([f(bl[..., :, 1:], (-1,)), br], -1)
    return 0.25 * torch.cat([top, bot], -2)


def _strip_weights(pairs):
    """Linear maps of a 15x15 surface to the two strip rows: [P][30][225], NaN rows as a mask [P][30]."""
    w, bad = np.zeros((len(pairs), 30, 225)), np.zeros((len(pairs), 30), bool)
    for p, (_, _, kind, _, bx, by) in enumerate(pairs):
        for e in range(30):
            row, sc = e // 15, e % 15 - 7
            for down in ((-1,) if row == 0 else (-1, 1)):
                if kind < 2:
                    a, b = sc + 0.5 * (row & 1), 0.5 * down * row
                    x, y = (a, b) if kind == 0 else (b, a)
                elif kind < 4:
                    x, y = sc - ((down * row) >> 1), sc + ((down * row + 1) >> 1)
                    y = y if kind == 2 else -y
                else:
                    bx32, by32, a, b = np.float32(bx), np.float32(by), np.float32(sc + 0.5 * (row & 1)), np.float32(0.5 * down * row)
                    x, y = float(a) * float(bx32) - float(b) * float(by32), float(a) * float(by32) + float(b) * float(bx32)
                if abs(x) > 7 or abs(y) > 7:
                    bad[p, e] = True
                    continue
                x0, y0 = min(int(math.floor(x + 7)), 13), min(int(math.floor(y + 7)), 13)
                dx, dy = x + 7 - x0, y + 7 - y0
                for oy, wy in ((0, 1 - dy), (1, dy)):
                    for ox, wx in ((0, 1 - dx), (1, dx)):
                        w[p, e, (y0 + oy) * 15 + x0 + ox] += wx * wy * (1.0 if row == 0 else 0.5)
    return _t(w), torch.tensor(bad, device="cuda")


def _half_window(n, hwidth, blur, scale):
    i = np.arange(n, dtype=float)
    w = np.where(i < hwidth - blur / 2, 1.0, np.where(i > hwidth + blur / 2, 0.0, 0.5 * (1 - np.sin(np.pi * (i - hwidth) / blur))))
    return w * scale / (w[0] + 2 * w[1:].sum())


def _centroid_weights():
    """Weights and doubled offsets of the windowed centroid for each integer maximum: [15][30] each."""
    wy, wx = _half_window(2, 1.0, 1.0, 1.0), _half_window(9, 6.0, 5.0, 2.0)
    w, x = np.zeros((15, 30)), np.zeros((15, 30))
    for i in range(15):
        for dy in range(2):
            for adx in range(9):
                for s in ((1,) if adx == 0 else (-1, 1)):
                    if (adx - dy) & 1:
                        continue
                    k = (adx * s) >> 1
                    if 0 <= i + k < 15:
                        w[i, dy * 15 + i + k] = (1.0 if dy == 0 else 2.0) * wy[dy] * wx[adx]
                        x[i, dy * 15 + i + k] = 2 * k + dy
    return _t(w), _t(x)


def _extract(corr, pairs, strips, centroid):
    """Disparity records [n][9] of the surfaces."""
    n = corr.shape[0]
    w, bad = strips
    v = torch.einsum("pec,npc->npe", w, corr.reshape(n, -1, 225)) + _OFFSET
    pos = (v > 0).all(1)
    combo = torch.where(pos, torch.exp(torch.log(torch.where(v > 0, v, torch.ones_like(v))).mean(1)) - _OFFSET, torch.zeros_like(v[:, 0]))
    nan = bad.any(0)
    row0 = torch.where(nan[:15], torch.full_like(combo[:, :15], -math.inf), combo[:, :15])
    ix = row0.argmax(1)
    vmax = combo.gather(1, ix[:, None])[:, 0]
    cw, cx = centroid[0][ix], centroid[1][ix]
    m = torch.where((combo > 0) & ~nan, combo, torch.zeros_like(combo)) * cw
    s0, sx = m.sum(1), (m * cx).sum(1)
    ok = vmax >= _MIN_CORR
    nanv, zero, fx = torch.full_like(s0, math.nan), torch.zeros_like(s0), (ix - 7).to(_F)
    has = ok & (s0 != 0)
    cm = -(fx + sx / torch.where(s0 != 0, s0, torch.ones_like(s0)) / 2)
    rec = [torch.where(ok, -fx, nanv), torch.where(has, cm, nanv), torch.where(ok, vmax, zero)]
    for kind in (0, 1):
        idx = [i for i, p in enumerate(pairs) if p[2] == kind]
        if not idx:
            rec += [nanv, zero]
            continue
        s = corr[:, idx] if kind == 0 else corr[:, idx].transpose(-1, -2)
        p = (0.5 * (s + torch.flip(s, (-2,))) + _OFFSET).prod(1)
        p = torch.where(p > 0, p.clamp_min(0) ** (1.0 / len(idx)), torch.zeros_like(p)) - _OFFSET
        i = torch.arange(15, device=corr.device)
        notch = torch.where((i < 6) | (i > 8), torch.sin(math.pi * (i + 1).to(_F) / 16), torch.zeros(15, dtype=_F, device=corr.device))
        prof = torch.einsum("nij,i->nj", p, notch)
        ic = prof.argmax(1)
        f0, f1, f2 = (prof.gather(1, (ic + k).clamp(0, 14)[:, None])[:, 0] for k in (-1, 0, 1))
        den = f0 - 2 * f1 + f2
        xc = ic + torch.where((ic > 0) & (ic < 14) & (den != 0), 0.5 * (f0 - f2) / torch.where(den != 0, den, torch.ones_like(den)), zero)
        ir = torch.floor(xc + 0.5).long().clamp(0, 14)
        rec += [-(xc - 7), prof.gather(1, ir[:, None])[:, 0] / 8]
    return torch.stack(rec + [torch.where(has, s0, nanv), torch.where(ok, fx, nanv)], 1)


def _imclt(sc, case, tab, clt, tiles, frames):
    """Adds the inverse transforms of the tiles to frames [S][C][H + 8][W + 8]."""
    W = case["width"]
    lpf = 0.25 * sc["lpf"].cuda().to(_F).reshape(-1, 1, 8, 8)
    t = clt * lpf
    blk = 0
    for m in range(4):
        blk = blk + torch.einsum("yv,nschv,xh->nscyx", tab["inv"][m >> 1], t[:, :, :, m], tab["inv"][m & 1])
    tx = W // 8
    at = ((tiles // tx) * 8 * (W + 8) + (tiles % tx) * 8)[:, None] + (torch.arange(16, device="cuda")[:, None] * (W + 8) + torch.arange(16, device="cuda")[None]).reshape(1, -1)
    S, C = frames.shape[:2]
    frames.view(S, C, -1).index_add_(2, at.reshape(-1), blk.permute(1, 2, 0, 3, 4).reshape(S, C, -1))


def _exact_scene(case, seed):
    sc, tab = _scene(case, seed), _dtt_tables()
    W, H, S, C, use = case["width"], case["height"], case["sensors"], case["colors"], case["use"]
    T = (W // 8) * (H // 8)
    lpf, strips, cen = _corr_lpf(tab), _strip_weights(sc["pairs"]), _centroid_weights()
    rec = torch.full((T, 9), math.nan, dtype=_F, device="cuda")
    rec[:, [2, 4, 6]] = 0
    frames = torch.zeros((S, C, H + 8, W + 8), dtype=_F, device="cuda") if use in ("frame", "render") else None
    chosen = torch.nonzero(sc["op"])[:, 0]
    step = max(16, 60000 // (S * C + 4 * len(sc["pairs"])))
    grads = None
    if use == "adjoint":
        grads = {"grad_extrinsics": torch.zeros((S, 4), dtype=_F, device="cuda"), "grad_disparity": torch.zeros(T, dtype=_F, device="cuda"),
                 "jac_extrinsics": torch.zeros((T, S, 4), dtype=_F, device="cuda"), "jac_disparity": torch.zeros(T, dtype=_F, device="cuda"),
                 "disparity": torch.full((T,), math.nan, dtype=_F, device="cuda")}
    g = sc["geometry"]
    for t in chosen.split(step):
        if use == "adjoint":
            e = torch.stack([_t(g[k]) for k in ("azimuth", "tilt", "roll", "zoom")], -1)[None].repeat(len(t), 1, 1).requires_grad_()
            ports, d = _ports(sc, case, t, e, sc["target"][t].to(_F).requires_grad_())
        else:
            ports, d = _ports(sc, case, t)
            if use == "render":  # the tasks carry their ports in 32 bits
                ports = ports.float().to(_F)
        clt = _clt(sc, case, tab, ports)
        if frames is not None:
            _imclt(sc, case, tab, clt, t, frames)
        if use == "render":
            continue
        r = _extract(_corr(clt, tab, lpf, sc["pairs"]), sc["pairs"], strips, cen)
        if grads is None:
            rec[t] = r
            continue
        cm = r[:, 1]
        ok = torch.isfinite(cm)
        je, jd = torch.autograd.grad(torch.where(ok, cm, torch.zeros_like(cm)).sum(), (e, d))
        cm = torch.where(ok, cm, torch.zeros_like(cm)).detach()
        grads["disparity"][t] = r[:, 1].detach()
        grads["jac_extrinsics"][t], grads["jac_disparity"][t] = je, jd
        grads["grad_disparity"][t] = 2 * cm * jd
        grads["grad_extrinsics"] += (2 * cm[:, None, None] * je).sum(0)
    if use == "adjoint":
        return grads
    if use == "render":
        return list(frames)
    return [rec] + list(frames) if use == "frame" else rec


def exact(case, seed):
    if case["use"] in ("lma", "texture"):  # iterated fits; per-pixel choices between near ties
        return None
    if case["use"] == "batch":
        return [_exact_scene(case, seed * 64 + i) for i in range(case["scenes"])]
    return _exact_scene(case, seed)
