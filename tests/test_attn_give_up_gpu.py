"""Attention kernels whose waits for copies run out at once (TG_ATTN_POLLS=0): the call returns an error, and the next ones the bits that they
returned before. In a cluster the first CTA has to stay until the others, which give their copies time to land, have handed over."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one cluster per cache with idle CTAs, every CTA at work, no clusters; caches of which a warp takes several groups of keys, more than its ring holds
@pytest.mark.parametrize("n,S", [(3, 61), (8, 250), (9, 61), (2, 300), (3, 700), (70, 250)])
def test_batched_step(capi, synth, weights_270m, monkeypatch, n, S):
    m = capi.Model("270m").load_file(weights_270m).build_tables(1024)
    prompts = np.stack([synth.random_prompt(S, 50 + i) for i in range(n)])
    step = synth.random_prompt(n, 9)

    def logits(give_up):
        st = m.state(n, S + 8)
        st.prefill(prompts, want_logits=False)
        try:
            if not give_up:
                return st.decode(step).copy()
            monkeypatch.setenv("TG_ATTN_POLLS", "0")
            with pytest.raises(capi.TgError) as e:
                st.decode(step)
            assert e.value.code == capi.TG_ECUDA and "wait ran out" in str(e.value)
        finally:
            monkeypatch.delenv("TG_ATTN_POLLS", raising=False)
            st.close()

    want = logits(False)
    logits(True)
    assert np.array_equal(logits(False), want) and np.all(np.isfinite(want))
    m.close()


# CUDA cores: walks of one CTA, of a cluster, and more steps than the ring holds; tensor cores: windows that begin in the first and in a later key tile
@pytest.mark.parametrize("S", [24, 61, 178, 500, 941, 1500])
def test_prompt(capi, synth, weights_270m, monkeypatch, S):
    m = capi.Model("270m").load_file(weights_270m).build_tables(1024)
    ids, st = synth.random_prompt(S, 3), m.state(1, S + 8)
    want = st.prefill(ids)
    st.reset()
    monkeypatch.setenv("TG_ATTN_POLLS", "0")
    with pytest.raises(capi.TgError) as e:
        st.prefill(ids)
    assert e.value.code == capi.TG_ECUDA and "wait ran out" in str(e.value)
    monkeypatch.delenv("TG_ATTN_POLLS")
    st.reset()
    assert np.array_equal(st.prefill(ids), want) and np.all(np.isfinite(want))
    st.close()
    m.close()
