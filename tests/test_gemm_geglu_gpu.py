"""up | gate multiplied in the GEMM's epilogue (many rows) against the raw sums and a GeGLU kernel (few): prompts of a small group get
the bits they get alone, where the rows together pass the line between the two and alone do not. Row counts that end inside a group of 8
tokens and a tile of 64, tables in shared memory with steps of a power of two and of none, and one too large for shared memory."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,n,S,table", [("1B", 2, 303, 1024), ("1B", 2, 480, 1000), ("1B", 2, 500, 2049), ("270m", 2, 959, 1024),
                                            ("270m", 2, 901, 2048), ("270m", 2, 1200, 1 << 16)])
def test_group_keeps_the_bits(capi, synth, weights_270m, weights_1b, size, n, S, table):
    m = capi.Model(size).load_file(weights_270m if size == "270m" else weights_1b)
    m.build_tables(table)
    prompts = np.stack([synth.random_prompt(S, 360 + i) for i in range(n)])
    st, one = m.state(n, S + 8), m.state(1, S + 8)
    logits = st.prefill(prompts)
    for i in range(n):
        one.reset()
        assert np.array_equal(logits[i], one.prefill(prompts[i])[0]), i
    for x in (st, one, m):
        x.close()
