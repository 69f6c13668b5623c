"""The min-p sampler of one sequence, spread over all CTAs: its token against the sequential fp32 running sum over the
very probabilities that it wrote (a flat, an ordinary and a steep row, crossings from the first to the last column), and
the same uniforms through the device loop."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("temp", [0.05, 0.7, 50.0])
def test_grid_minp_is_the_sequential_crossing(capi, synth, weights_270m, temp):
    m = capi.Model("270m").load_file(weights_270m)
    m.build_tables(1024)
    st = m.state(1, 64)
    prompt = synth.random_prompt(9, 5)
    for r in (0.0, 1e-6, 0.004, 0.03, 0.25, 0.5, 0.77, 0.999, 1.5):
        st.reset()
        st.prefill(prompt, want_logits=False)
        tok = int(st.sample_minp(0.1, temp, np.float32([r]))[0])
        p = st.logits()[0]
        hit = np.nonzero(np.cumsum(p, dtype=np.float32) >= np.float32(r))[0]  # (numpy adds one after the other)
        assert tok == (hit[0] if hit.size else 0), r
        rf = np.float32([0.1, r, 0.6, r])
        st.reset()
        st.prefill(prompt, want_logits=False)
        loop = st.generate([tok], 4, 0.1, temp, rf).reshape(-1)
        st.reset()
        st.prefill(prompt, want_logits=False)
        feed, steps = np.int32([tok]), []
        for x in rf:
            st.decode(feed, want_logits=False)
            feed = st.sample_minp(0.1, temp, np.float32([x])).astype(np.int32)
            steps.append(int(feed[0]))
        assert loop.tolist() == steps, r
    st.close()
    m.close()
