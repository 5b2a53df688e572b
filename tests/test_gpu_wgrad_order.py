"""GPU: the order of the weight gradient's FP32 sums. The tensor core's accumulator truncates,
so a gradient element depends on how its products are divided into chains: another division
moves the gradient by 1e-5 and more at 128^3, and a training run with it. tests/golden/
wgrad_order.npz holds up to 4096 elements of every convolution's weight gradient, from the
library as of commit 73410b6 (tests/golden/make_wgrad_order.py). What may differ is the order of
the at most 148 atomic additions per element that join the chains: sqrt(148) 2^-24 = 7e-7 of an
element's larger partial sums; 2e-6 per tensor leaves a factor for sums that cancel."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "wgrad_order.npz")
SHAPE = (64, 100, 128)


def step_inputs():
    """Parameters, input fields and target from numpy's generator alone."""
    import unet_ref as R

    rng = np.random.default_rng(31)
    lay, total = R.layout()
    flat = np.zeros(total, dtype=np.float32)
    for k, (o, shp) in lay.items():
        n = int(np.prod(shp))
        fan = {"up2.w": 64, "up1.w": 32, "out.w": 16}.get(k, 27 * shp[1] if len(shp) == 5 else 1)
        flat[o:o + n] = rng.standard_normal(n) * (np.sqrt(2.0 / fan) if k.endswith(".w") else 0.05)
    x = (rng.standard_normal((1, 4) + SHAPE) * 0.5 + 0.3).astype(np.float32)
    t = (rng.standard_normal((1,) + SHAPE) * 0.1).astype(np.float32)
    return flat, x, t


def samples(grads):
    """Up to 4096 elements of every convolution's weight gradient."""
    import unet_ref as R

    lay, _ = R.layout()
    out = {}
    for k, (o, shp) in lay.items():
        if len(shp) == 5:
            n = int(np.prod(shp))
            at = np.sort(np.random.default_rng(n + o).choice(n, min(n, 4096), replace=False))
            out[k] = grads[o + at]
    return out


def test_weight_gradient_keeps_its_chains(pkg, ctx):
    flat, x, t = step_inputs()
    with pkg.UNet(ctx, seed=1) as net:
        net.set_params(flat)
        got = samples(net.train_step(x, t, lr=0.0, want_grads=True)[1])
    with np.load(GOLDEN) as want:
        off = {k: np.linalg.norm(got[k].astype(np.float64) - want[k]) / np.linalg.norm(want[k].astype(np.float64))
               for k in got}
    assert max(off.values()) <= 2e-6, off
