"""Scores that overflow to -inf weigh nothing, however many of them stand together: a softmax over the whole row gives them probability 0.
One layer without rotation; the last token's query meets keys whose product with it is -1.6e51, and its own, which gives 0."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A, B = 0, 1  # the token whose key repels, and the one whose query is repelled


def small_model(capi, synth, monkeypatch):
    c = synth.Config(640, 2048, 1, 8192, 1024, 512, 256, 4, 1, 1_000_000.0, 10_000.0, 6)
    monkeypatch.setitem(synth.CONFIGS, "one layer", c)
    rng = np.random.default_rng(2)
    t = {}
    for name, kind, shape, off in synth.layout("one layer"):
        t[name] = rng.integers(-127, 128, shape, dtype=np.int8) if kind == "i1" else np.full(shape, 1 / 127 if name.endswith(".s") else 0.0, np.float32)
    del t["<end>"]
    t["wte.q"][[A, B]] = 0
    t["wte.q"][A, 0] = t["wte.q"][B, 1] = 127
    t["lm_head.q"] = np.ascontiguousarray(t["wte.q"].T)
    for p, at in (("q", [(1, 256 * h, 127) for h in range(4)]), ("k", [(0, 0, -127), (1, 5, 127)]), ("v", [(0, 7, 127), (1, 9, 127)])):
        t["l0.%s.q" % p][:] = 0
        for row, col, v in at:
            t["l0.%s.q" % p][row, col] = v
    for p in ("q", "k"):
        t["l0.%s_norm" % p][0] = 1e25
    blob = np.concatenate([x.reshape(-1).view(np.uint8) for x in t.values()])
    m = capi.Model.__new__(capi.Model)
    m.lib, m.size, m.h = capi.load(), "one layer", C.c_void_p()
    m.cfg = capi.tg_config(*[getattr(c, f) for f, _ in capi.tg_config._fields_])
    assert m.lib.tg_model_create(C.byref(m.cfg), 0, C.byref(m.h)) == 0
    m.load_bytes(blob).build_tables(1024)
    one, nil = np.ones((1024, 256), np.float32), np.zeros((1024, 256), np.float32)
    for local in (0, 1):
        assert m.lib.tg_model_set_rope(m.h, local, one.ctypes.data_as(C.c_void_p), nil.ctypes.data_as(C.c_void_p), 1024) == 0
    return m


# a step of a warp, a round of all warps, several, keys shared by a cluster
@pytest.mark.parametrize("S", [9, 24, 33, 61, 150])
def test_short_prompt(capi, synth, monkeypatch, S):
    m = small_model(capi, synth, monkeypatch)
    st = m.state(1, 256)
    got = st.prefill([A] * (S - 1) + [B])
    st.reset()
    want = st.prefill([B] * S)  # scores of 0: the mean of equal values
    st.close()
    m.close()
    assert np.all(np.isfinite(got))
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)  # fp32 sums in another order
