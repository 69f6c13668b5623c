"""The short-prompt attention with the keys of two queries shared by a cluster of CTAs, against the tensor-core kernel (every CTA walks
all keys): prompts on both sides of every change of the number of CTAs, whose last chunk of 32 keys and last pair of queries are
full or not, and turns behind a context, where up to six CTAs share them."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctx,S", [(0, 96), (0, 97), (0, 127), (0, 128), (0, 129), (0, 178), (0, 191), (0, 193), (700, 33), (700, 61), (1500, 47)])
def test_shared_keys(capi, synth, weights_270m, monkeypatch, ctx, S):
    m = capi.Model("270m").load_file(weights_270m)
    m.build_tables(1 << 20)
    st = m.state(1, 2048)
    ids = synth.random_prompt(ctx + S, 7)
    got = []
    for split in (True, False):
        st.reset()
        if ctx:
            st.prefill(ids[:ctx], want_logits=False)
            if split:
                got.append(st.append(ids[ctx:]))
            else:  # the same tokens one by one
                for t in ids[ctx:-1]:
                    st.decode([int(t)], want_logits=False)
                got.append(st.decode([int(ids[-1])]))
        else:
            monkeypatch.setenv("TG_ATTN_SMALL_MAX", "960" if split else "1")
            got.append(st.prefill(ids))
    st.close()
    m.close()
    # fp32 softmax sums in another order, 18 layers: the bound of the other comparisons of attention kernels
    assert rel_l2(got[0], got[1]) <= 1e-4, (ctx, S)
    assert np.all(np.isfinite(got[0]))


@pytest.mark.parametrize("n,S", [(1, 672), (1, 673), (4, 170), (5, 150), (5, 151), (20, 61), (21, 61),
                                 (1, 832), (1, 833), (4, 177), (4, 178), (22, 61)])  # rows 832; 400 + 55000 / S
def test_line_between_the_kernels(capi, synth, weights_270m, monkeypatch, n, S):
    """Prompts and groups on both sides of the line between the attention kernels, against the short-prompt kernel."""
    m = capi.Model("270m").load_file(weights_270m)
    m.build_tables(1 << 20)
    prompts = np.stack([synth.random_prompt(S, 20 + i) for i in range(n)])
    st = m.state(n, S + 8)
    a = st.prefill(prompts)
    st.reset()
    monkeypatch.setenv("TG_ATTN_SMALL_MAX", "100000")
    b = st.prefill(prompts)
    st.close()
    m.close()
    for i in range(n):
        assert rel_l2(a[i], b[i]) <= 5e-5, i
