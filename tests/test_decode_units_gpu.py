"""The decode kernel's units are refilled for the next layer while their columns leave: one launch of many tokens and one launch per
token (other kernels in between) give the same bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,prompt", [("270m", 5), ("270m", 530), ("1B", 40)])
def test_one_launch_equals_a_launch_per_token(capi, synth, request, size, prompt):
    m = capi.Model(size).load_file(request.getfixturevalue("weights_" + size.lower())).build_tables()
    ids, steps = synth.random_prompt(prompt, 1), 48
    rf = synth.mt19937_uniforms(steps, 5)
    hidden, toks = [], []
    for single in (False, True):
        st = m.state(1, prompt + steps + 2)
        st.prefill(ids, want_logits=False)
        t = [st.sample_argmax()]
        if single:
            for i in range(steps):
                st.decode(t[-1])
                t.append(st.sample_minp(0.1, 0.7, rf[i : i + 1]))
        else:
            t += list(st.generate(t[0], steps, 0.1, 0.7, rf))
        toks.append(np.concatenate([np.ravel(x) for x in t]))
        hidden.append(st.hidden())
        st.close()
    m.close()
    assert np.array_equal(toks[0], toks[1])
    assert np.array_equal(hidden[0], hidden[1])
