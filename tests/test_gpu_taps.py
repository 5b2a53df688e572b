"""GPU: the register-window passes of 7, 9, 13 and 17 taps (and a support that keeps the loop
over taps) against the oracle: the filter on volumes shorter than, as long as and longer than
the windows and tiles, zero and periodic boundary, FP64 1e-13 and FP32 2e-6 (the bounds of
test_gpu_ops.py); and a segmentation whose every pass has 13 taps, or 13 along k only, FP64
1e-9, FP32 1e-5 (the bounds of test_gpu_rsfe.py)."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cyclic", [False, True])
@pytest.mark.parametrize("sigma, h", [(1.0, (1.0, 1.0, 1.0)), (2.0, (1.0, 1.0, 1.0)), (2.0, (1.0, 1.0, 1.5)),
                                      (4.0, (1.0, 1.0, 1.5)), (1.5, (1.0, 1.0, 1.0))])
@pytest.mark.parametrize("shape", [(3, 4, 5), (13, 7, 9), (20, 66, 130), (67, 5, 33), (9, 65, 129)])
def test_filter(ctx, O, shape, sigma, h, cyclic):
    x = np.random.default_rng(sum(shape)).random(shape)
    want = O.gauss_filter(x, sigma, h=h, cyclic=cyclic)
    assert rel(ctx.gauss_filter(x, sigma, h=h, cyclic=cyclic), want) < 1e-13
    assert rel(ctx.gauss_filter(x.astype(np.float32), sigma, h=h, cyclic=cyclic), want) < 2e-6


@pytest.mark.parametrize("sigma, h", [(2.0, (1.0, 1.0, 1.0)), (3.0, (1.0, 1.0, 1.5)), (4.0, (1.0, 1.0, 1.5))])
@pytest.mark.parametrize("shape", [(20, 22, 24), (35, 18, 33)])
def test_segmentation(pkg, ctx, O, shape, sigma, h):
    u0 = pkg.synth.ellipsoids(shape, 3, n=2, semi_axes=(4, 7))
    phi0 = pkg.synth.sphere_phi0(shape, 6.0)
    kw = dict(sigma=sigma, lamda1=1.0, lamda2=1.2, epsilon=1e-3, lamda=0.5, maxiter=4, ls_steps=1, tol=0.0,
              bc=pkg.BC_NEU, gs_rel_res_tol=1e-8)
    want = O.rsfe_apply(u0, phi0, O.default_params(**kw), h=h)
    got = ctx.rsfe_apply(u0, phi0, pkg.default_params(**kw), h=h, want_u=True, want_f=True)
    for key in ("phi", "u", "f1", "f2"):
        assert rel(got[key], want[key]) <= 1e-9, key
    kw["gs_rel_res_tol"] = 1e-6
    want = O.rsfe_apply(u0, phi0, O.default_params(**kw), h=h)
    got = ctx.rsfe_apply(u0.astype(np.float32), phi0.astype(np.float32), pkg.default_params(**kw), h=h, want_u=True,
                         want_f=True)
    for key in ("u", "f1", "f2"):
        assert rel(got[key], want[key]) <= 1e-5, key
