"""GPU: the general half-sweep (rb_half_vec_kernel: own value, omega) with and without the FP64
divisions: spacings and time steps that are powers of two, or not, or mixed. Red-black sweeps
with the own value: bit-exact against the oracle. Solves with omega 1.4, where the oracle adds
u_in / dt after b (one rounding per update apart): 1e-13."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bc_type, bc", [("dir", 0.0), ("dir", 0.3), ("neu", 0.0), ("neu", 0.3)])
@pytest.mark.parametrize("h, dt", [((1.0, 1.0, 1.0), 1.0), ((1.0, 0.5, 2.0), 0.7), ((0.7, 1.0, 1.5), 1.0),
                                   ((0.7, 1.1, 1.5), 0.8)])
@pytest.mark.parametrize("shape", [(3, 3, 3), (5, 6, 7), (9, 7, 17), (33, 20, 18), (8, 33, 64)])
def test_general_half_sweeps(pkg, ctx, O, shape, h, dt, bc_type, bc):
    rng = np.random.default_rng(sum(shape))
    u = rng.standard_normal(shape)
    b = rng.standard_normal(shape)
    kw = dict(dt=dt, bc=bc, bc_type=pkg.BC_NEU if bc_type == "neu" else pkg.BC_DIR, h=h)
    want = O.poisson_sweeps(u, b, order=pkg.SWEEP_REDBLACK, sweeps=3, **kw)
    got = u.copy()
    ctx.poisson_sweeps(got, b, order=pkg.SWEEP_REDBLACK, sweeps=3, **kw)
    assert np.array_equal(got, want)
    kw.update(tol=1e-30, max_sweeps=5, check_every=5, omega=1.4)
    got = u.copy()
    ctx.poisson_solve(got, b, **kw)
    assert rel(got, O.poisson_solve(u, b, **kw)[0]) <= 1e-13
