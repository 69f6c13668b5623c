"""The integer GEMM with every number of ring stages (few tokens: many small ones) against float64: K of fewer, as many and more stages than
the ring has, the line of 64 tokens up to which single CTAs take a tile, columns enough for many tiles per CTA. Exact digit sums: bound 2e-7 as in test_gemm_i8_gpu."""

import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 8, 9, 24, 33, 48, 57, 64, 65])
@pytest.mark.parametrize("K,N", [(1152, 1024), (6912, 640), (640, 262144)])
def test_ring(capi, M, K, N):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randint(-128, 128, (K, N), dtype=torch.int8, device="cuda", generator=g)
    s = torch.rand(N, device="cuda", generator=g) * 1e-2 + 1e-4
    c = torch.full((M, N), float("nan"), device="cuda")
    torch.cuda.synchronize()
    assert capi.load().tg_dev_qgemm(*[C.c_void_p(t.data_ptr()) for t in (c, x, w, s)], M, K, N, None) == 0
    for n in range(0, N, 65536):
        want = (x.double() @ w[:, n:n + 65536].double()) * s[n:n + 65536].double()
        assert float((c[:, n:n + 65536].double() - want).norm() / want.norm()) <= 2e-7, n
