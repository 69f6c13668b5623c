"""The integer GEMM around the line between its two rings: eight small stages for tiles of one or two token groups (up to 16 rows), four stages of eight groups
above, with both epilogues. Sums against float64 at the bound of test_gemm_i8_gpu; the arg-max epilogue against the logits of single steps."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [7, 15, 16, 17, 23, 25])
@pytest.mark.parametrize("K,N", [(640, 1024), (1152, 6912), (6912, 1152), (1152, 262144)])
def test_sums(capi, M, K, N):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(100 + M)
    x = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randint(-128, 128, (K, N), dtype=torch.int8, device="cuda", generator=g)
    s = torch.rand(N, device="cuda", generator=g) * 1e-2 + 1e-4
    c = torch.full((M, N), float("nan"), device="cuda")
    torch.cuda.synchronize()
    assert capi.load().tg_dev_qgemm(*[C.c_void_p(t.data_ptr()) for t in (c, x, w, s)], M, K, N, None) == 0
    for n in range(0, N, 65536):
        want = (x.double() @ w[:, n:n + 65536].double()) * s[n:n + 65536].double()
        assert float((c[:, n:n + 65536].double() - want).norm() / want.norm()) <= 2e-7, n


@pytest.mark.parametrize("n", [8, 15, 16, 17, 24, 25])
def test_arg_max(capi, synth, weights_270m, n):
    m = capi.Model("270m").load_file(weights_270m).build_tables(1024)
    prompts = np.stack([synth.random_prompt(4, 190 + i) for i in range(n)])
    one, run = m.state(n, 32), m.state(n, 32)
    for st in (one, run):
        st.prefill(prompts, want_logits=False)
    tok = first = one.sample_argmax()
    steps = []
    for _ in range(4):
        tok = one.generate(tok, 1)[0]
        assert np.array_equal(tok, one.logits().argmax(axis=1))
        steps.append(tok)
    assert np.array_equal(run.generate(first, 4), np.stack(steps))
    for x in (one, run, m):
        x.close()
