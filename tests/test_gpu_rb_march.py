"""GPU: the half-sweep of the residual solve (rb_march_kernel) against red-black sweeps on
b_eff = b + u_in / dt restated in numpy with the kernel's operations.

A solve that stops at a sweep cap is a fixed number of sweeps. FP64: bit-exact. FP32: each
update rounds a few times (relative 2^-24 each) and the sweep contracts errors, so k sweeps
stay within a few 1e-7 of FP64: bound 1e-6. The restatement is held to the FP64 oracle, which
adds u_in / dt after b (one rounding per update apart): 1e-13.
Sizes: the smallest volume, rows shorter and longer than a vector group, odd and even
rows with and without padding, plane counts around the planes per thread, and thin volumes
of many planes, which take the larger number of planes per thread.
"""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (4, 5, 7), (5, 4, 8), (7, 6, 9), (6, 9, 16), (9, 7, 17), (8, 33, 31), (13, 5, 64),
          (3560, 5, 9), (4740, 4, 10)]


def _sweeps(u, b, h, dt, bc, neu, count):
    u = u.copy()
    shape = u.shape
    pos = np.indices(shape)
    face = [(pos[a] == 0) | (pos[a] == shape[a] - 1) for a in range(3)]
    nb = sum(f.astype(int) for f in face)
    if not neu:
        u[nb > 0] = bc
    beff = b + u * (1.0 / dt)
    diag = 1.0 / dt
    for a in range(3):
        diag = diag + (np.where(face[a], 1.0, 2.0) if neu else 2.0) / (h[a] * h[a])
    ht = 1.0 / diag
    bcn = np.array([bc, bc, (1.0 / np.sqrt(2.0)) * bc, (1.0 / np.sqrt(3.0)) * bc])[nb]
    for _ in range(count):
        for color in (0, 1):
            terms = []
            for a in range(3):
                lo = np.concatenate([np.zeros_like(u.take([0], a)), u.take(range(shape[a] - 1), a)], a)
                hi = np.concatenate([u.take(range(1, shape[a]), a), np.zeros_like(u.take([0], a))], a)
                lo = np.where(pos[a] == 0, -(bcn * h[a]), lo)
                hi = np.where(pos[a] == shape[a] - 1, bcn * h[a], hi)
                terms.append((lo + hi) / (h[a] * h[a]))
            v = (terms[0] + terms[1] + terms[2] + beff) * ht
            upd = (pos.sum(0) + color) % 2 == 0
            u = np.where(upd & ((nb == 0) | neu), v, u)
    return u


@pytest.mark.parametrize("bc_type, bc", [("dir", 0.0), ("dir", 0.3), ("neu", 0.0), ("neu", 0.3)])
@pytest.mark.parametrize("h", [(1.0, 1.0, 1.0), (0.7, 1.0, 1.5)])
@pytest.mark.parametrize("shape", SHAPES)
def test_half_sweeps(pkg, ctx, O, shape, h, bc_type, bc):
    rng = np.random.default_rng(shape[0] + 7 * shape[2])
    u = rng.standard_normal(shape)
    b = rng.standard_normal(shape)
    neu = bc_type == "neu"
    kw = dict(dt=0.8, bc=bc, bc_type=pkg.BC_NEU if neu else pkg.BC_DIR, tol=1e-30, max_sweeps=5, check_every=5, h=h)
    want = _sweeps(u, b, h, 0.8, bc, neu, 5)
    assert rel(want, O.poisson_solve(u, b, **kw)[0]) <= 1e-13
    got = u.copy()
    ctx.poisson_solve(got, b, **kw)
    assert np.array_equal(got, want)
    got32 = u.astype(np.float32)
    ctx.poisson_solve(got32, b.astype(np.float32), **kw)
    assert rel(got32, want) <= 1e-6
