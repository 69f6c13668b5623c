"""Decode steps of several sequences against the same sequences one by one (the batch-1 step has an attention of its
own): contexts around the edges of a warp's 4 keys, a round of 32 keys and the ring of a sliding-window layer, with one
split of the cache and with many."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S", [(2, 1), (3, 3), (2, 28), (150, 31), (40, 33), (3, 64), (2, 509), (5, 511), (2, 700)])
def test_batched_step_is_each_sequence(capi, synth, weights_270m, n, S):
    m = capi.Model("270m").load_file(weights_270m)
    m.build_tables(1 << 20)
    prompts = np.stack([synth.random_prompt(S, 70 + i) for i in range(n)])
    steps = np.stack([synth.random_prompt(n, 90 + i) for i in range(4)])
    st, one = m.state(n, S + 16), m.state(1, S + 16)
    st.prefill(prompts, want_logits=False)
    logits = [st.decode([int(t) for t in row]).copy() for row in steps]
    for i in sorted({0, n // 2, n - 1}):
        one.reset()
        one.prefill(prompts[i], want_logits=False)
        for row, lg in zip(steps, logits):
            assert rel_l2(lg[i], one.decode([int(row[i])])[0]) <= 1e-4, i
    st.close()
    one.close()
    m.close()
