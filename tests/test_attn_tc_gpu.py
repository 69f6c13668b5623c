"""The tensor-core attention keeps a row's result apart from keys that the row may not see."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOKEN, DIM = 4711, 17


@pytest.fixture(scope="module")
def outlier_blob(synth, weights_270m):
    """The 270m weights with a dimension of the embedding that only one token uses; its gain in the first layer's norm is left to
    the test."""
    lay = {name: (shape, off) for name, _, shape, off in synth.layout("270m")}
    blob = np.fromfile(weights_270m, np.uint8)
    (V, D), off = lay["wte.q"]
    wte = blob[off:off + V * D].view(np.int8).reshape(V, D)
    wte[:, DIM] = 0
    wte[TOKEN, DIM] = 127
    off = lay["l0.attn_pre"][1]
    return blob, blob[off:off + 4 * D].view(np.float32)


# |v| of the last token hundreds of times that of the others; infinite
@pytest.mark.parametrize("gain", [1e3, 3e38])
def test_a_later_value_changes_no_earlier_row(capi, synth, outlier_blob, gain):
    blob, norm = outlier_blob
    norm[DIM] = gain
    m = capi.Model("270m").load_bytes(blob).build_tables(1024)
    S, slots = 1100, 512
    st = m.state(1, 1152)
    ids = synth.random_prompt(S, 5)
    rows = (S - 1) // 64 * 64  # 64 keys are worked on together: a probability of 0 times infinity is NaN in the last token's tile
    got = []
    for last in (int(ids[0]), TOKEN):
        ids[-1] = last
        st.reset()
        st.prefill(ids, want_logits=False)
        got.append([x[:rows] for x in st.kv_read(5, 0, S)] + [x[:rows - (S - slots)] for x in st.kv_read(1, 0, slots)])
    st.close()
    m.close()
    for a, b in zip(*got):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)


def test_gains_and_values_of_wide_range(capi, synth, weights_270m, monkeypatch):
    """Norm gains of q and k and columns of v that differ by up to 2^10, against the fp32 kernels."""
    lay = {name: (shape, off) for name, _, shape, off in synth.layout("270m")}
    blob = np.fromfile(weights_270m, np.uint8)
    rng = np.random.default_rng(3)
    for name, (shape, off) in lay.items():
        if name.endswith((".q_norm", ".k_norm", ".v.s")):
            f = blob[off:off + 4 * shape[0]].view(np.float32)
            wide = np.exp2(-rng.uniform(0, 10, shape[0])).astype(np.float32)
            f[:] = f * wide if name.endswith(".v.s") else (1 + f) * wide - 1  # (a norm's gain is 1 + w)
    m = capi.Model("270m").load_bytes(blob).build_tables(1 << 20)
    st = m.state(1, 1152)
    ids = synth.random_prompt(1100, 6)
    got = []
    for tc in ("1", "0"):
        monkeypatch.setenv("TG_ATTN_TC", tc)
        st.reset()
        logits = st.prefill(ids)
        got.append((logits,) + st.kv_read(5, 0, 1100) + st.kv_read(17, 0, 1100))
    st.close()
    m.close()
    for a, b in zip(*got):
        assert rel_l2(a, b) <= 5e-5  # (the bound of the other comparisons of attention kernels)
