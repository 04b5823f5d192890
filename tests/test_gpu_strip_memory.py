"""The strip products that a forward hands to its extraction pass lie in the room that the combined strip leaves; only
strips of more than 8 rows need a buffer of their own.  Under a memory limit that leaves no room for it the correlation
set-up is accepted all the same and the general kernels run, with the same results."""
import ctypes as C

import numpy as np
import pytest

from helpers import make_gpu
from tileproc import _lib as L
from tileproc import synth

pytestmark = pytest.mark.gpu


def _usage(tp):
    n = C.c_size_t()
    assert tp._lib.tp_get_memory_usage(tp.h, C.byref(n)) == L.TP_OK
    return n.value


@pytest.mark.parametrize("kind", ["quad_mono", "quad_bayer"])
def test_long_strips_under_a_memory_limit(kind):
    w, h = 72, 40
    sc = synth.make_scene(kind, seed=95, width=w, height=h)
    T = (w // 8) * (h // 8)
    kw = {"corr_strip_hight": 16, "corr_wndy_size": 16}
    lib = L.load()
    out = []
    try:
        for limited in (False, True):
            with make_gpu(sc) as tp:
                tp.setCorrelation()
                used = _usage(tp)
                tp.setCorrelation(corr_strip_hight=8, corr_wndy_size=8)
                assert _usage(tp) == used
                if limited:
                    lib.tp_set_memory_limit(used)
                tp.setCorrelation(**kw)
                assert _usage(tp) == used + (0 if limited else T * 240 * 4)
                tp.setFullFrameImages(np.full(T, 3.0, np.float32))
                tp.process()
                out.append((tp.getClt(), tp.getCorr(), tp.getDisparity()))
                tp.setCorrelation()
                tp.process()
                out[-1] += (tp.getDisparity(),)
                lib.tp_set_memory_limit(0)
    finally:
        lib.tp_set_memory_limit(0)
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True)
