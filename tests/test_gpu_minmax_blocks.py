"""GPU: the minimum and maximum behind the component's pivot at counts around a block's and a
grid's share (one value per thread, a short last round, several rounds), with the extremes in
the first and in the last cell. The component is the whole numbers 0 and 1: bit for bit the
oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 8, 8), (5, 7, 33), (3, 5, 64), (70, 90, 97)])
@pytest.mark.parametrize("low_first", [True, False])
def test_component_with_extremes_at_the_ends(ctx, O, dtype, shape, low_first):
    x = np.random.default_rng(sum(shape)).uniform(-1, 1, shape).astype(dtype)
    x.flat[0], x.flat[-1] = (-5, 7) if low_first else (7, -5)
    ijk = tuple(n // 2 for n in shape)
    for threshold in (0.4, 0.5):
        got = ctx.connected_component(x, ijk=ijk, threshold=threshold)
        want = O.connected_component(x.astype(np.float64), ijk=ijk, threshold=threshold)
        assert np.array_equal(got, want)
