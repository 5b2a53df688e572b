"""GPU: the divergence of column kernels (planes in groups, faces by selects) and its spacings on
volumes whose plane count leaves a short last group, shorter and longer than a block along k:
FP64 bit for bit the oracle's; FP32 within the rounding of its terms (each one-sided term sums
8 |v| <= 8 in at most 4 roundings and the sum of three terms has 2 more, so 8 units of 2^-24 on
8 (1/2hx + 1/2hy + 1/2hz))."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [(1.0, 1.0, 1.0), (0.7, 0.5, 1.3)])
@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 5, 6), (5, 3, 67), (7, 18, 131), (6, 9, 64)])
def test_div(ctx, O, shape, h):
    v = np.random.default_rng(sum(shape)).uniform(-1, 1, (3,) + shape)
    v = v.astype(np.float32).astype(np.float64)
    want = O.div(v, h)
    assert np.array_equal(ctx.div(v, h), want)
    got = ctx.div(v.astype(np.float32), h)
    terms = 8.0 * sum(1.0 / (2.0 * a) for a in h)
    # the low x face ends in "/ 2 * hx"
    terms = max(terms, 8.0 * (h[0] / 2.0 + sum(1.0 / (2.0 * a) for a in h[1:])))
    assert np.abs(got - want).max() <= 8 * 2.0 ** -24 * terms
