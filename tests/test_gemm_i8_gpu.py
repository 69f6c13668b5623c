"""The integer tensor-core GEMM (kernels_gemm_i8.cuh) at the edges of its tiles: token groups of 8, tiles of 64 tokens
and 128 columns, K-splits, the longest K; and rows that a shared exponent could spoil. Compared with float64: the digit
sums are exact, so what is left is one fp32 rounding per join (relative L2 about 5e-8; bound 2e-7)."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def case(M, K, N, seed=3):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((M, K)).astype(np.float32)
    w = rng.integers(-128, 128, (K, N), dtype=np.int8)
    s = (rng.random(N, dtype=np.float32) * 1e-2 + 1e-4).astype(np.float32)
    return x, w, s


def exact(x, w, s):
    return (x.astype(np.float64) @ w.astype(np.float64)) * s.astype(np.float64)


@pytest.mark.parametrize("M", [1, 7, 8, 9, 63, 64, 65, 129, 513])
@pytest.mark.parametrize("K,N", [(256, 256), (640, 1152), (6912, 640)])
def test_tile_edges(capi, M, K, N):
    x, w, s = case(M, K, N)
    assert rel_l2(capi.qgemm(x, w, s), exact(x, w, s)) <= 2e-7


def test_many_tiles_per_cta(capi):
    # 54 column tiles x 33 token tiles: twelve tiles per CTA, both accumulators reused
    x, w, s = case(2051, 256, 6912)
    assert rel_l2(capi.qgemm(x, w, s), exact(x, w, s)) <= 2e-7


def test_more_tiles_than_a_16_bit_square(capi):
    # 4360 rows of the vocabulary's columns: the tile index times its divisor passes 2^32 (70656 tiles of one CTA)
    import ctypes as C

    torch = pytest.importorskip("torch")
    M, K, N = 4360, 256, 262144
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randint(-128, 128, (K, N), dtype=torch.int8, device="cuda", generator=g)
    s = torch.rand(N, device="cuda", generator=g) * 1e-2 + 1e-4
    c = torch.full((M, N), float("nan"), device="cuda")
    torch.cuda.synchronize()
    args = [C.c_void_p(t.data_ptr()) for t in (c, x, w, s)]
    assert capi.load().tg_dev_qgemm(*args, M, K, N, None) == 0
    torch.cuda.synchronize()
    for n in range(0, N, 32768):
        want = (x.double() @ w[:, n:n + 32768].double()) * s[n:n + 32768].double()
        err = (c[:, n:n + 32768].double() - want).norm() / want.norm()
        assert float(err) <= 2e-7, n


def test_rows_of_any_range(capi):
    x, w, s = case(12, 1152, 640)
    x[1] *= 1e-30                    # tiny and huge rows beside ordinary ones: the exponent is per row
    x[2] *= 1e25
    x[3] = 0
    x[4] *= np.exp(3 * np.random.default_rng(1).standard_normal(1152)).astype(np.float32)  # six decades inside a row
    x[5] = np.float32(2.0) ** np.arange(1152, dtype=np.float32).clip(0, 20)               # powers of two: the top of the range
    x[6] = 1.0 - 2.0 ** -24
    x[7, 5] = np.nan
    x[8, 6] = np.inf
    c = capi.qgemm(x, w, s)
    want = exact(np.where(np.isfinite(x), x, 0), w, s)
    for r in (0, 1, 2, 4, 5, 6, 9, 10, 11):
        assert rel_l2(c[r], want[r]) <= 2e-7, r
    assert not c[3].any()
    assert np.isnan(c[7]).all() and not np.isfinite(c[8]).any()


@pytest.mark.parametrize("K,N", [(256, 640), (1152, 256), (2048, 256), (6912, 1152)])
@pytest.mark.parametrize("M", [1, 9, 130])
def test_columns_that_do_not_see_the_large_elements(capi, K, N, M):
    """every third row holds a few elements far above the rest, which half of the columns give the weight 0: these columns
    are sums of the others alone, and keep fp32's precision however large the few are (the exponent of a row's digits is the
    largest element's). Bound per row: 24-bit inputs and one rounding, 2^-24 each; rows of ordinary range 2e-7 as above."""
    x, w, s = case(M, K, N)
    big = [0, K // 2, K - 1]
    for i, r in enumerate(range(0, M, 3)):
        x[r, big] = np.float32(10.0) ** (4 + 2 * (i % 8)) * np.float32([1.0, -0.7, 0.3])
    w[big, ::2] = 0
    c = capi.qgemm(x, w, s)
    want = exact(x, w, s)
    for r in range(M):
        assert rel_l2(c[r, ::2], want[r, ::2]) <= 2e-7, r
        assert rel_l2(c[r, 1::2], want[r, 1::2]) <= 2e-7, r
    x *= np.float32(2.0 ** -112)  # rows near the end of fp32's range
    s *= np.float32(2.0 ** 100)
    c, want = capi.qgemm(x, w, s), exact(x, w, s)
    for r in range(M):
        assert rel_l2(c[r], want[r]) <= 2e-7, r


def test_wide_rows_in_a_captured_graph(capi):
    """a replay looks at the rows that it finds: ordinary ones when the graph is captured, wide ones when it is replayed"""
    import ctypes as C

    torch = pytest.importorskip("torch")
    M, K, N = 40, 1152, 640
    x, w, s = case(M, K, N)
    xd, wd, sd = (torch.from_numpy(t).cuda() for t in (x, w, s))
    c = torch.empty(M, N, device="cuda")
    stream = torch.cuda.Stream()
    args = [C.c_void_p(t.data_ptr()) for t in (c, xd, wd, sd)] + [M, K, N, C.c_void_p(stream.cuda_stream)]
    lib = capi.load()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        assert lib.tg_dev_qgemm(*args) == 0  # (the scratch is there before the capture)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            assert lib.tg_dev_qgemm(*args) == 0
    x[5, 7] = 1e9
    w[7, :] = 0
    xd.copy_(torch.from_numpy(x))
    wd.copy_(torch.from_numpy(w))
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    got, want = c.cpu().numpy(), exact(x, w, s)
    for r in range(M):
        assert rel_l2(got[r], want[r]) <= 2e-7, r


@pytest.mark.parametrize("K,N", [(640, 1024), (2048, 1152), (1152, 6912)])
def test_captured_matvec_keeps_its_bits(capi, K, N):
    """small matrices are launched without the programmatic edge inside a graph, larger ones with it; each node follows
    the kernel that writes its input"""
    import ctypes as C

    torch = pytest.importorskip("torch")
    x, w, s = case(8, K, N)
    xd, wd, sd = (torch.from_numpy(t).cuda() for t in (x, w, s))
    y, xi = torch.empty(8, N, device="cuda"), torch.empty(K, device="cuda")
    lib, stream = capi.load(), torch.cuda.Stream()

    def call(i):
        xi.copy_(xd[i])
        assert lib.tg_dev_qmatvec(*[C.c_void_p(t.data_ptr()) for t in (y[i], xi, wd, sd)], K, N, C.c_void_p(stream.cuda_stream)) == 0

    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        call(0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for i in range(8):
                call(i)
    y.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    for i in range(8):
        assert np.array_equal(y[i].cpu().numpy(), capi.qmatvec(x[i], w, s)), i
