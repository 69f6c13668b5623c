"""The vocabulary matvec's ring over every depth it accepts, against fp64."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

N = 262144


@pytest.mark.parametrize("K", [256, 640, 1024, 1152, 2048, 6912])
def test_every_depth(capi, K):
    g = torch.Generator(device="cuda").manual_seed(K)
    x = torch.randn(K, device="cuda", generator=g)
    w = torch.randint(-127, 128, (K, N), dtype=torch.int8, device="cuda", generator=g)
    s = torch.rand(N, device="cuda", generator=g) + 0.1
    y = torch.empty(N, device="cuda")
    p = [C.c_void_p(t.data_ptr()) for t in (y, x, w, s)]
    assert capi.load().tg_dev_qmatvec(*p, K, N, C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want = torch.cat([x.double() @ w[:, c:c + 16384].double() for c in range(0, N, 16384)]) * s.double()
    # a row set adds K / 4 terms, rounded by up to 2^-25 of a partial sum that grows like the root of its length: about
    # sqrt(K) / 6 * 2^-24 of the result, 8e-7 at 6912; six times that
    assert float((y.double() - want).norm() / want.norm()) <= 5e-6
