"""The attention kernels at the edges of their tiles, against kernels of another construction. 270m weights, a GeLU table of 2^20 entries: what
is left is fp32 sums in another order over 18 layers, the bound of the other comparisons of attention kernels."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def model(capi, weights):
    m = capi.Model("270m").load_file(weights)
    return m.build_tables(1 << 20)


# tensor cores: query tiles of 32 and key tiles of 128 that end inside, windows that begin in every quarter of a key tile, one and
# several K-splits of the projections, prompts of a group
@pytest.mark.parametrize("n,S", [(1, 24), (1, 127), (1, 128), (1, 129), (1, 161), (1, 513), (1, 545), (1, 640), (1, 737), (1, 1025), (1, 2050), (5, 33), (6, 97), (4, 641)])
def test_tensor_cores_against_cuda_cores(capi, synth, weights_270m, monkeypatch, n, S):
    m = model(capi, weights_270m)
    st = m.state(n, S + 8)
    prompts = np.stack([synth.random_prompt(S, 500 + i) for i in range(n)])
    got = []
    for small_up_to in ("1", "1000000"):
        monkeypatch.setenv("TG_ATTN_SMALL_MAX", small_up_to)
        st.reset()
        logits = st.prefill(prompts)
        rows = min(S, 512)
        got.append([logits] + [x for i in sorted({0, n - 1}) for layer in (0, 17) for x in st.kv_read(layer, 0, rows if layer == 0 else S, i)])
    st.close()
    m.close()
    for a, b in zip(*got):
        assert rel_l2(a, b) <= 5e-5 and np.all(np.isfinite(a))


# CUDA cores: clusters of every size with shared and with own walks, none, odd numbers of pairs, the last CTA of a cluster without work
@pytest.mark.parametrize("ctx,S", [(0, 1), (0, 3), (0, 65), (0, 126), (0, 150), (0, 195), (0, 196), (0, 221), (0, 940), (0, 941), (40, 90), (900, 33), (1500, 61), (1500, 65), (1500, 101)])
def test_shared_and_own_walks(capi, synth, weights_270m, monkeypatch, ctx, S):
    m = model(capi, weights_270m)
    st = m.state(1, 2048)
    ids = synth.random_prompt(ctx + S, 11)
    if ctx:
        st.prefill(ids[:ctx], want_logits=False)
        a = st.append(ids[ctx:])
        st.reset()
        st.prefill(ids[:ctx], want_logits=False)
        for t in ids[ctx:-1]:
            st.decode([int(t)], want_logits=False)
        b = st.decode([int(ids[-1])])
    else:
        a = st.prefill(ids)
        st.reset()
        monkeypatch.setenv("TG_GEMM_TC", "0")  # GEMMs and attention of their own
        b = st.prefill(ids)
    st.close()
    m.close()
    assert rel_l2(a, b) <= 1e-4 and np.all(np.isfinite(a))


# a batch's step: one and several clusters per cache, their last CTAs idle, the line of 8 sequences, caches read evict-first
@pytest.mark.parametrize("n,S", [(2, 255), (3, 256), (3, 257), (8, 300), (9, 300), (2, 1100), (4, 1500), (70, 250)])
def test_batched_step(capi, synth, weights_270m, n, S):
    m = model(capi, weights_270m)
    prompts = np.stack([synth.random_prompt(S, 70 + i) for i in range(n)])
    steps = np.stack([synth.random_prompt(n, 90 + i) for i in range(3)])
    st, one = m.state(n, S + 16), m.state(1, S + 16)
    st.prefill(prompts, want_logits=False)
    logits = [st.decode([int(t) for t in row]).copy() for row in steps]
    for i in sorted({0, n - 1}):
        one.reset()
        one.prefill(prompts[i], want_logits=False)
        for row, lg in zip(steps, logits):
            assert rel_l2(lg[i], one.decode([int(row[i])])[0]) <= 1e-4, i
    for x in (st, one, m):
        x.close()
