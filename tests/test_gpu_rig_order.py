"""tp_rig_correlate reads the auxiliary camera's CLT and tile map on the main camera's stream or a caller's, and
returns at once.  A setter or forward of the auxiliary camera called next waits for it: the rig's record equals that
of the same call read back before the auxiliary camera is touched again, bit for bit.  Forwards of the main camera
are enqueued before the rig call, so that the auxiliary camera's calls land before the rig's kernel has run."""
import ctypes as C

import numpy as np
import pytest

from helpers import make_gpu
from tileproc import synth

pytestmark = pytest.mark.gpu

W, H = 648, 488
T = (W // 8) * (H // 8)


@pytest.mark.parametrize("own_stream", [False, True])
def test_aux_setters_wait_for_the_rig(own_stream):
    import torch
    sc = synth.make_scene("quad_mono", seed=29, width=W, height=H)
    aux = dict(sc)
    aux["images"] = np.ascontiguousarray(np.roll(sc["images"], 2, axis=-1))
    disp = np.full(T, 2.0, np.float32)
    first = np.ones(T, np.int32)
    first[::7] = 0
    nxt = np.zeros(T, np.int32)  # the next list names other tiles only
    nxt[::7] = 1
    with make_gpu(sc) as tm, make_gpu(aux) as ta:
        stream = torch.cuda.Stream()
        sp = None if own_stream else C.c_void_p(stream.cuda_stream)
        for tp in (tm, ta):
            tp.setCorrelation()
        tm.setFullFrameImages(disp)
        ta.setFullFrameImages(disp, tile_op=first)
        tm.process()
        ta.process()
        corr0, rec0 = tm.rigCorrelate(ta)
        assert np.isnan(rec0[::7, 0]).all() and np.isfinite(rec0[first != 0, 0]).any()
        for _ in range(3):
            ta.setFullFrameImages(disp, tile_op=first)
            ta.process()
            for _ in range(40):
                tm._ck(tm._lib.tp_process(tm.h, sp), "tp_process")
            tm._ck(tm._lib.tp_rig_correlate(tm.h, ta.h, C.c_float(0.55), 0, sp), "tp_rig_correlate")
            ta.setFullFrameImages(disp + 1, tile_op=nxt)
            ta.process()
            corr, rec = np.zeros_like(corr0), np.zeros_like(rec0)
            tm._ck(tm._lib.tp_get_rig(tm.h, corr.ctypes.data_as(C.c_void_p), rec.ctypes.data_as(C.c_void_p)),
                   "tp_get_rig")
            assert np.array_equal(rec, rec0, equal_nan=True)
            assert np.array_equal(corr[first != 0], corr0[first != 0], equal_nan=True)
        torch.cuda.synchronize()
