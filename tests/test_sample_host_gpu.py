"""Sampling from host logits with the result in memory of its own: arrays of any layout, against the call in place, bit for bit."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["plain", "read-only", "2-d", "fortran", "strided", "float64", "unaligned"])
def test_result_apart_from_the_logits(capi, form):
    base = np.random.default_rng(5).normal(0, 3, 16384).astype(np.float32)
    x = {"plain": base, "read-only": base, "2-d": base.reshape(128, 128), "fortran": np.asfortranarray(base.reshape(128, 128)), "float64": base.astype(np.float64),
         "strided": np.repeat(base, 2)[::2], "unaligned": np.frombuffer(b"x" + base.tobytes(), np.float32, offset=1)}[form]
    if form == "read-only":
        x.setflags(write=False)
    before = x.copy()
    tok, p = capi.minp_logits(x, 0.1, 0.7, 0.4)
    q = np.array(x, np.float32, copy=True)
    t = C.c_int(-1)
    assert capi.load().tg_minp_logits(q.ctypes.data_as(C.c_void_p), q.size, 0.1, 0.7, 0.4, C.byref(t)) == 0
    assert tok == t.value and p.shape == x.shape and p.dtype == np.float32 and p.flags.writeable
    assert np.array_equal(p, q) and np.array_equal(x, before)
