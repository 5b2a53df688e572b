"""GPU: the convolution's entry point (Context.conv3d_bf16) against FP64 convolutions of the same
BF16 numbers: 1e-5 relative, the order of the FP32 sums (as in test_gpu_unet.py)."""
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _inputs(seed, dims=(6, 8, 32), cin=16, cout=32):
    gen = torch.Generator().manual_seed(seed)
    x = torch.randn((1,) + dims + (cin,), generator=gen).to(torch.bfloat16)
    w = (torch.randn((cout, cin, 3, 3, 3), generator=gen) * 0.2).to(torch.bfloat16).float()
    return x, w, torch.randn(cout, generator=gen)


def _want(x, w, b):
    return torch.nn.functional.conv3d(x.double().permute(0, 4, 1, 2, 3), w.double(), b.double(),
                                      padding=1).permute(0, 2, 3, 4, 1).numpy()


def test_inputs_written_on_a_side_stream(ctx):
    """x, w and bias are still being written on torch's current stream when the call is made."""
    x, w, b = _inputs(1)
    xd, wd, bd = x.cuda(), w.cuda(), b.cuda()
    x2, w2, b2 = torch.zeros_like(xd), torch.zeros_like(wd), torch.zeros_like(bd)
    ctx.conv3d_bf16(xd, wd, bd)  # the context's workspace exists
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)  # about 10 ms of clock cycles before the copies
        x2.copy_(xd)
        w2.copy_(wd)
        b2.copy_(bd)
        got = ctx.conv3d_bf16(x2, w2, b2)
    assert rel(got.cpu().double().numpy(), _want(x, w, b)) <= 1e-5


@pytest.mark.parametrize("nz", [24, 144])
def test_refused_width_leaves_nothing_running(pkg, nz):
    """A width without a tiling is refused, and nothing queued by the call still reads its
    arguments: the context's stream, busy before the call, is idle after it."""
    x, w, b = (t.cuda() for t in _inputs(2, dims=(3, 4, nz)))
    with pkg.Context(0) as c:
        stream = torch.cuda.Stream()
        c.set_stream(stream.cuda_stream)
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)  # about 10 ms of clock cycles
        with pytest.raises(pkg.Im3dError):
            c.conv3d_bf16(x, w, b)
        assert stream.query()
        c.set_stream(None)


@pytest.mark.parametrize("cout, dims", [(32, (3, 6, 112)), (64, (6, 12, 128)), (32, (2, 5, 256)), (64, (9, 3, 96))])
def test_64_channels_on_wide_rows(ctx, cout, dims):
    """64 staged channels and 32 outputs per block leave room for one tile row only on rows of
    112 and more."""
    x, w, b = _inputs(3, dims=dims, cin=64, cout=cout)
    got = ctx.conv3d_bf16(x.cuda(), w, b)
    assert rel(got.cpu().double().numpy(), _want(x, w, b)) <= 1e-5
