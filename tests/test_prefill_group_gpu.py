"""Equal prompts prefilled together against each of them alone, on both sides of the line between the attention kernels
of short prompts and of many rows, with lengths that end inside a tile of 32 queries and of 64 keys (the GEMMs see other
row counts, so the logits agree to rounding)."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S", [(2, 479), (2, 481), (31, 31), (31, 33), (5, 193), (13, 95), (2, 961), (256, 4),
                                 (123, 16), (128, 16), (300, 15), (45, 33), (47, 33), (970, 1),
                                 (239, 16), (240, 16), (62, 33), (63, 33)])  # a group's line: 400 + 55000 / S rows, S >= 16
def test_group_is_each_prompt(capi, synth, weights_270m, n, S):
    m = capi.Model("270m").load_file(weights_270m)
    m.build_tables(1 << 20)
    prompts = np.stack([synth.random_prompt(S, 40 + i) for i in range(n)])
    st, one = m.state(n, S + 8), m.state(1, S + 8)
    logits = st.prefill(prompts)
    for i in sorted({0, 1, n // 2, n - 1}):
        one.reset()
        assert rel_l2(logits[i], one.prefill(prompts[i])[0]) <= 5e-5, i
    st.close()
    one.close()
    m.close()


def test_small_batch_keeps_the_bits_of_one_prompt(capi, synth, weights_270m):
    """Two prompts whose rows together, but not alone, pass the line between the attention kernels."""
    m = capi.Model("270m").load_file(weights_270m)
    m.build_tables(1024)
    prompts = np.stack([synth.random_prompt(490, 60 + i) for i in range(2)])
    st, one = m.state(2, 512), m.state(1, 512)
    logits = st.prefill(prompts)
    for i in range(2):
        one.reset()
        assert np.array_equal(logits[i], one.prefill(prompts[i])[0]), i
    st.close()
    one.close()
    m.close()


@pytest.mark.parametrize("n,S", [(4, 148), (4, 149), (7, 211)])
def test_group_of_the_larger_model(capi, synth, weights_1b, n, S):
    """Rows of 6912 columns on both sides of the line from which the GEMM multiplies up and gate itself (4 per SM)."""
    m = capi.Model("1B").load_file(weights_1b)
    m.build_tables(1 << 20)
    prompts = np.stack([synth.random_prompt(S, 80 + i) for i in range(n)])
    st, one = m.state(n, S + 8), m.state(1, S + 8)
    logits = st.prefill(prompts)
    for i in (0, n - 1):
        one.reset()
        assert rel_l2(logits[i], one.prefill(prompts[i])[0]) <= 5e-5, i
    st.close()
    one.close()
    m.close()
