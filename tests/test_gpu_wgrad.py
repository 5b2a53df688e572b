"""GPU: the weight gradient where its plan has edges: rows past the last tile, units that end
inside the volume, more planes than the rings hold, the tile widths 16 to 128 of the three
levels. The gradient of two samples is the mean of their own gradients: every activation and
data gradient is the same BF16 number up to the factor 2 of the mean, and the weight gradients
add the same products in other units and blocks. The FP32 accumulators may truncate at each of
up to a few hundred additions per block (2^-24 each): 2e-5 relative per parameter tensor. The
single-sample gradients are held to the network on the CPU in test_gpu_unet.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")


@pytest.mark.parametrize("shape", [(44, 4, 64), (4, 28, 64), (12, 12, 128), (4, 4, 256), (20, 36, 64)])
def test_two_samples_are_the_mean(pkg, ctx, shape):
    import unet_ref as R

    rng = np.random.default_rng(sum(shape))
    net = pkg.UNet(ctx, seed=9)
    flat = net.get_params()
    lay, _ = R.layout()
    o, _ = lay["out.w"]
    flat[o:o + 16] = rng.standard_normal(16) * 0.3
    x = rng.standard_normal((2, 4) + shape).astype(np.float32)
    t = rng.standard_normal((2,) + shape).astype(np.float32)
    with net:
        net.set_params(flat)
        both = net.train_step(x, t, lr=0.0, want_grads=True)[1].astype(np.float64)
        one = [net.train_step(x[q:q + 1], t[q:q + 1], lr=0.0, want_grads=True)[1].astype(np.float64) for q in (0, 1)]
    mean = (one[0] + one[1]) / 2
    for k, (o, shp) in lay.items():
        n = int(np.prod(shp))
        a, b = both[o:o + n], mean[o:o + n]
        assert np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(b), k
