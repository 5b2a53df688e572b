"""GPU: connected components on words of 32 cells against the oracle, bit-exact: rows shorter
than a word, of exactly one, one cell more, of several; tiles that end inside the volume; 2-D
images; both connectivities; white faces (which receive but do not spread); a component that
runs along words through many tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(5, 6, 7), (9, 17, 32), (18, 5, 33), (17, 18, 64), (33, 20, 65), (4, 40, 130), (3, 3, 3), (40, 70, 1),
          (17, 33, 2)]


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("density", [0.35, 0.6])
def test_components_of_noise(ctx, O, shape, full, density):
    rng = np.random.default_rng(shape[0] * 100 + shape[2] + int(10 * density))
    x = (rng.random(shape) < density).astype(np.float64)
    x[0, 0, 0], x[-1, -1, -1] = 0.0, 1.0
    inner = [p for p in np.argwhere(x > 0) if all(1 <= c <= n - 2 for c, n in zip(p, shape) if n > 2)]
    ijk = tuple(int(c) for c in inner[len(inner) // 2]) if inner else (1, 1, 0)
    want = O.connected_component(x, ijk, full_connected=full)
    assert np.array_equal(ctx.connected_component(x, ijk, full_connected=full), want)
    got32 = ctx.connected_component(x.astype(np.float32), ijk, full_connected=full)
    assert np.array_equal(got32, want.astype(np.float32))
    init = (rng.random(shape) < 0.02).astype(np.float64)
    want = O.connected_component(x, init=init, full_connected=full, binary_output=False)
    assert np.array_equal(ctx.connected_component(x, init=init, full_connected=full, binary_output=False), want)


def test_a_path_along_words(ctx, O):
    x = np.zeros((6, 40, 200))
    for r in range(1, 38):  # rows joined at alternating ends
        x[2, r, 1:199] = 1.0 if r % 2 else 0.0
        if r % 2 == 0:
            x[2, r, 198 if (r // 2) % 2 else 1] = 1.0
    want = O.connected_component(x, (2, 1, 5))
    assert want.sum() > 3000
    assert np.array_equal(ctx.connected_component(x, (2, 1, 5)), want)
