"""GPU: every gradient of a training step against FP64 sums over the same BF16 activations and
gradients (plain torch on the CUDA device in float64, tests/unet_ref.py).

The network is built so that no activation and no data gradient depends on the order of a sum:
every output channel of a convolution has one tap of weight 1 (a random one of 27, from one input
channel), likewise every child and channel of the transposed convolutions; the inputs and the
output layer's weights are positive BF16 numbers of few exponents, and the target is the
prediction minus a BF16 number. All values the GPU rounds are then known to the bit, all sums
have positive terms, and what remains are the gradients' own FP32 sums:

* convolutions' filters: chains of L multiplications on the tensor core, whose accumulator loses
  less than 2^-23 of itself at each, then at most 148 rounded atomics: (L + 16) 2^-23.
* transposed convolutions' filters: 4 multiplications per chain (4 x 2^-23), then rounded
  additions, a few hundred of them with random errors of 2^-24: 1.6e-6.
* biases and the output layer: rounded additions, some thousands by atomics: 1e-5.

A wrong tap, a dropped row or plane, or a tile counted twice moves an element by 1e-3 and more.
Shapes: rows past the last tile of 8, 4, 2 rows, every tile width, two samples, chains of several
tiles (up to 12 at 64 x 100 x 64, with 96 rows through rings of 8 and 5)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def routed_network(rng):
    import unet_ref as R

    lay, total = R.layout()
    flat = np.zeros(total, dtype=np.float32)
    for name, cin, cout in R.CONV:
        o, shp = lay[name + ".w"]
        w = np.zeros((cout, cin, 27), dtype=np.float32)
        used = 4 if name == "e1a" else cin
        src = np.concatenate([rng.permutation(used) for _ in range(-(-cout // used))])[:cout]
        w[np.arange(cout), src, rng.integers(0, 27, cout)] = 1
        flat[o:o + w.size] = w.ravel()
    for name, cin, cout in (("up2", 64, 32), ("up1", 32, 16)):
        o, shp = lay[name + ".w"]
        w = np.zeros(shp, dtype=np.float32)
        for c in range(8):
            w[c, rng.permutation(cin)[:cout], np.arange(cout)] = 1
        flat[o:o + w.size] = w.ravel()
    o, _ = lay["out.w"]
    flat[o:o + 16] = 2.0 ** -(np.arange(16) % 3)
    return flat, lay


def bound(name, shp, nsamp, dims):
    if name.endswith(".w") and len(shp) == 5:
        level = 0 if name[:2] in ("e1", "d1") else 1 if name[:2] in ("e2", "d2") else 2
        D, H, W = (d >> level for d in dims)
        chains = -(-148 // (shp[1] // 16))
        # tiles of at most 8 rows of at most 128 voxels: an even share and one tile more
        L = nsamp * D * H * W / 16 / chains + 8 * min(W, 128) / 16
        return (L + 16) * 2.0 ** -23
    return 1.6e-6 if name in ("up1.w", "up2.w") else 1e-5


@pytest.mark.parametrize("nsamp, dims", [(1, (64, 100, 64)), (2, (20, 36, 64)), (1, (12, 28, 128)), (1, (8, 12, 256)),
                                         (2, (128, 128, 256))])
def test_gradients_are_the_sums(pkg, ctx, nsamp, dims):
    import unet_ref as R

    rng = np.random.default_rng(sum(dims) + nsamp)
    flat, lay = routed_network(rng)
    gen = torch.Generator(device="cuda").manual_seed(sum(dims))
    # inputs 1 .. 1.99 in steps of 2^-7, and 1 .. 1.98 in steps of 2^-6 for the loss's differences
    x = 1 + torch.randint(0, 128, (nsamp, 4) + dims, generator=gen, device="cuda").float() / 128
    m = 1 + torch.randint(0, 64, (nsamp,) + dims, generator=gen, device="cuda").float() / 64
    # (cuDNN may choose transforms, which leave 1e-16 where a value is exactly 0 or a BF16 number;
    # the plain product has one term per value; it needs 27 copies of the input)
    with torch.device("cuda"), torch.backends.cudnn.flags(enabled=m.numel() > 1 << 21):
        ps = {k: v.double().requires_grad_() for k, v in R.unflatten(flat).items()}
        y = R.forward(x.double(), ps, emulate_bf16=True, hooks=True)[:, 0]
        target = (y.detach() - m).float()
        assert torch.equal(target.double(), y.detach() - m)  # exact in FP32
        dy = 2 * m * (torch.ones(()) / torch.tensor(float(m.numel())))  # the kernel's FP32 operations
        y.backward(dy.double())
    torch.cuda.synchronize()
    with pkg.UNet(ctx, seed=1) as net:
        net.set_params(flat)
        loss, g = net.train_step(x, target, lr=0.0, want_grads=True)
    want_loss = float((m.double() ** 2).mean())
    assert abs(loss - want_loss) <= 1e-6 * want_loss
    for k, (o, shp) in lay.items():
        n = int(np.prod(shp))
        got = g[o:o + n].astype(np.float64)
        want = ps[k].grad.cpu().numpy().ravel()
        assert np.linalg.norm(want) > 0, k
        assert np.linalg.norm(got - want) <= bound(k, shp, nsamp, dims) * np.linalg.norm(want), (
            k, np.linalg.norm(got - want) / np.linalg.norm(want), bound(k, shp, nsamp, dims))
