"""tg_append of a longer turn (all tokens at once behind the cached context) against the same tokens fed one by one
through tg_decode (a key too many or too few moves the logits by percents): logits after the turn and after further steps, and the cache rows, for rings that are empty, partly
filled, full and wrapped, at the edges of the attention's two-query tiles and 32-key chunks."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctx,n", [(0, 32), (5, 33), (31, 64), (100, 61), (480, 65), (511, 32), (512, 47), (700, 130), (600, 600)])
def test_append_is_the_decode_of_its_tokens(capi, synth, weights_270m, ctx, n):
    m = capi.Model("270m").load_file(weights_270m)
    m.build_tables(1 << 20)
    prompt, turn, more = synth.random_prompt(max(ctx, 1), 3), synth.random_prompt(n, 4), synth.random_prompt(3, 5)
    a, b = m.state(1, 2048), m.state(1, 2048)
    for st in (a, b):
        if ctx:
            st.prefill(prompt, want_logits=False)
    if ctx >= 600:  # the ring goes on wrapping before the turn
        for t in more:
            for st in (a, b):
                st.decode([int(t)], want_logits=False)
    la = a.append(turn)
    for t in turn[:-1]:
        b.decode([int(t)], want_logits=False)
    lb = b.decode([int(turn[-1])])
    assert a.position() == b.position()
    assert rel_l2(la, lb) <= 1e-4
    for layer in (0, 5):  # a sliding-window and a global layer
        slots = 512 if layer == 0 else a.position()
        used = min(a.position(), slots)
        for x, y in zip(a.kv_read(layer, 0, used), b.kv_read(layer, 0, used)):
            assert rel_l2(x, y) <= 1e-4
    for t in more:
        assert rel_l2(a.decode([int(t)]), b.decode([int(t)])) <= 1e-4
    a.close()
    b.close()
    m.close()
