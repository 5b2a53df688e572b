"""GPU: the marching tensor-core convolution against an FP64 convolution of the same BF16
inputs and filter, where its plan has edges: more planes than TMEM slots and staged planes,
units that end inside the volume, rows past the last tile, every tile width, several units
per block and several samples. FP32 sums of up to 27 * 64 products whose order is fixed: 2e-6
relative (the accumulator may truncate: 108 additions of 2^-24 each, a quarter of that
measured on random signs)."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cin, cout, dims, nsamp", [
    (16, 16, (1, 1, 16), 1), (16, 16, (23, 19, 48), 1), (32, 32, (40, 9, 128), 1), (64, 64, (11, 13, 64), 2),
    (16, 32, (150, 5, 16), 1), (32, 16, (9, 33, 256), 1), (64, 32, (5, 3, 128), 1), (32, 64, (17, 70, 96), 3),
    (16, 16, (37, 130, 112), 1)])
def test_conv3d_march(ctx, cin, cout, dims, nsamp):
    gen = torch.Generator().manual_seed(cin + cout + sum(dims))
    x = torch.randn((nsamp,) + dims + (cin,), generator=gen).to(torch.bfloat16)
    w = (torch.randn((cout, cin, 3, 3, 3), generator=gen) * 0.2).to(torch.bfloat16).float()
    b = torch.randn(cout, generator=gen)
    got = ctx.conv3d_bf16(x.cuda(), w, b).cpu().double()
    want = torch.nn.functional.conv3d(x.double().permute(0, 4, 1, 2, 3), w.double(), b.double(), padding=1)
    assert rel(got.numpy(), want.permute(0, 2, 3, 4, 1).numpy()) <= 2e-6
