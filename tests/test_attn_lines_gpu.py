"""Which attention kernel a prompt or a group takes, just below and just above each line: the default call has the bits of the kernel that it should take and
not those of the other one, and both agree. A line that moves fails here until the cases move with it.

One prompt (or one of up to three): more than 940 tokens take the tensor cores. A group of n prompts of S tokens: n S > 700 + 50000 / S and S >= 24."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

CUDA_CORES = {"TG_ATTN_TC": "0"}
TENSOR_CORES = {"TG_ATTN_SMALL_MAX": "1", "TG_ATTN_TC_MIN": "1"}


def prefill(m, prompts, monkeypatch, env):
    with monkeypatch.context() as p:
        for k, v in env.items():
            p.setenv(k, v)
        st = m.state(len(prompts), prompts.shape[1] + 8)
        logits = st.prefill(prompts)
        st.close()
    return logits


@pytest.mark.parametrize("n,S,tensor_cores", [(1, 940, False), (1, 941, True), (3, 940, False), (2, 941, True),
                                              (4, 228, False), (4, 230, True),      # 912 of 919, 920 of 917 rows
                                              (24, 61, False), (25, 61, True),      # 1464, 1525 of 1519
                                              (34, 50, False), (35, 50, True),      # 1700, 1750 of 1700
                                              (115, 24, False), (116, 24, True),    # 2760, 2784 of 2783
                                              (200, 23, False)])
def test_kernel_of_a_prompt(capi, synth, weights_270m, monkeypatch, n, S, tensor_cores):
    m = capi.Model("270m").load_file(weights_270m).build_tables(1 << 20)
    prompts = np.stack([synth.random_prompt(S, 120 + i) for i in range(n)])
    got = prefill(m, prompts, monkeypatch, {})
    own, other = [prefill(m, prompts, monkeypatch, env) for env in ((TENSOR_CORES, CUDA_CORES) if tensor_cores else (CUDA_CORES, TENSOR_CORES))]
    m.close()
    assert np.array_equal(got, own) and not np.array_equal(got, other)
    for i in range(n):  # sums in another order, 18 layers: the bound of the other comparisons of attention kernels
        assert rel_l2(got[i], other[i]) <= 5e-5, i


# the short-prompt kernel against the long-prompt kernel of the CUDA cores: one to three CTAs share a walk, with walks of their own beside them or none, odd
# numbers of pairs, the last CTA of a cluster without work, walks that a window cuts
@pytest.mark.parametrize("S", [2, 3, 24, 32, 33, 64, 65, 95, 97, 126, 150, 195, 212, 213, 221, 513, 515, 940])
def test_short_prompt_kernel_against_the_long_prompt_kernel(capi, synth, weights_270m, monkeypatch, S):
    m = capi.Model("270m").load_file(weights_270m).build_tables(1 << 20)
    prompt = synth.random_prompt(S, 140)[None]
    a = prefill(m, prompt, monkeypatch, {})
    b = prefill(m, prompt, monkeypatch, {"TG_ATTN_TC": "0", "TG_ATTN_SMALL_MAX": "0"})
    m.close()
    assert not np.array_equal(a, b) or S < 4  # (another kernel; with a key or two its sums may be the same)
    assert rel_l2(a, b) <= 5e-5 and np.all(np.isfinite(a))
