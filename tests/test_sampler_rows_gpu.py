"""The row samplers (several CTAs per row): min-p's token against the sequential fp32 running sum over the very
probabilities it wrote, where segments are applied whole and where they are not; arg-max over several CTAs."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rows(kind, n, rng):
    if kind == "flat":
        return np.zeros(n, np.float32)
    if kind == "noise":
        return rng.standard_normal(n).astype(np.float32)
    if kind == "steep":  # a few tokens hold nearly everything: the sum jumps over many binades at once
        return rng.permutation(-4.0 * np.log1p(np.arange(n))).astype(np.float32)
    x = np.full(n, -300.0, np.float32)  # nearly all probabilities are zero
    x[rng.integers(0, n, 5)] = rng.standard_normal(5)
    return x


@pytest.mark.parametrize("n", [8192, 24576, 262144, 655360])
@pytest.mark.parametrize("kind", ["flat", "noise", "steep", "empty"])
def test_minp_token_is_the_sequential_crossing(capi, n, kind):
    rng = np.random.default_rng(n)
    x = rows(kind, n, rng)
    for r in (0.0, 1e-6, 0.03, 0.25, 0.5, 0.77, 0.999, 1.5):
        tok, p = capi.minp_logits(x, 0.1, 0.7, r)
        hit = np.nonzero(np.cumsum(p, dtype=np.float32) >= np.float32(r))[0]  # (numpy adds one after the other)
        assert tok == (hit[0] if hit.size else 0), r


@pytest.mark.parametrize("n", [4, 8188, 8196, 40000, 262144])
def test_argmax_over_parts(capi, n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal(n).astype(np.float32)
    for at in (0, n // 2, n - 1):
        y = x.copy()
        y[at:] = np.where(np.arange(n - at) % 3 == 0, np.float32(9.0), y[at:])  # the first of many equal maxima
        assert capi.argmax_logits(y) == at
    assert capi.argmax_logits(np.full(n, np.nan, np.float32)) == -1
    x[:] = -np.inf
    assert capi.argmax_logits(x) == -1
    x[n - 1], x[n - 2] = 0.0, -0.0
    assert capi.argmax_logits(x) == n - 2
