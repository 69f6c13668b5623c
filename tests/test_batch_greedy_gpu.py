"""Greedy runs of a batch: the steps before the last take each row's token from the keys that the vocabulary GEMM keeps, the last
one from the logits it leaves. One step per call always goes through the logits, so both give the same tokens and the same end."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S", [(2, 5), (9, 12), (64, 3), (130, 7), (300, 2)])
def test_a_run_of_steps_is_the_steps(capi, synth, weights_270m, n, S):
    m = capi.Model("270m").load_file(weights_270m)
    m.build_tables(1024)
    prompts = np.stack([synth.random_prompt(S, 170 + i) for i in range(n)])
    one, run = m.state(n, S + 32), m.state(n, S + 32)
    for st in (one, run):
        st.prefill(prompts, want_logits=False)
    tok = first = one.sample_argmax()
    steps = []
    for _ in range(9):
        tok = one.generate(tok, 1)[0]
        steps.append(tok)
        assert np.array_equal(tok, one.logits().argmax(axis=1))
    # runs of several lengths one after the other: eager steps, captured ones, and keys left clean between the two kinds
    got = [run.generate(first, 5)]
    got.append(run.generate(got[-1][-1], 3))
    got.append(run.generate(got[-1][-1], 1))
    assert np.array_equal(np.concatenate(got), np.stack(steps))
    assert np.array_equal(run.logits(), one.logits())
    for x in (one, run, m):
        x.close()
