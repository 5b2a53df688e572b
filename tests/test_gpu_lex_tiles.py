"""GPU: lexicographic sweeps by tiles (lex_tile_kernel) against the oracle's sequential
loops. FP64: bit-exact, whatever the number of tiles and of sweeps in one launch. FP32: a
few roundings of 2^-24 per update under a contraction: 1e-6 relative.
Sizes: below one tile, exactly one, one point more, ragged last tiles on each axis."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bc_type, bc", [("dir", 0.3), ("neu", 0.0), ("neu", 0.3)])
@pytest.mark.parametrize("shape, h, sweeps", [
    ((3, 3, 3), (1.0, 1.0, 1.0), 4), ((16, 16, 16), (1.0, 1.0, 1.0), 3), ((18, 18, 18), (0.8, 1.1, 1.3), 3),
    ((19, 17, 35), (1.0, 1.0, 1.0), 5), ((33, 34, 16), (0.5, 1.0, 2.0), 1), ((50, 3, 49), (1.0, 1.0, 1.5), 7),
    ((40, 52, 65), (1.0, 1.0, 1.0), 12)])
def test_lexicographic_tiles(pkg, ctx, O, shape, h, sweeps, bc_type, bc):
    rng = np.random.default_rng(sum(shape))
    u = rng.standard_normal(shape)
    b = rng.standard_normal(shape)
    kw = dict(dt=0.7, bc=bc, bc_type=pkg.BC_NEU if bc_type == "neu" else pkg.BC_DIR, sweeps=sweeps, h=h)
    want = O.poisson_sweeps(u, b, **kw)
    got = u.copy()
    ctx.poisson_sweeps(got, b, **kw)
    assert np.array_equal(got, want)
    got32 = u.astype(np.float32)
    ctx.poisson_sweeps(got32, b.astype(np.float32), **kw)
    assert rel(got32, want) <= 1e-6
