"""GPU: the sweeps of a small volume in one cluster (rb_cluster_kernel), against the numpy
restatement of test_gpu_rb_march.py: FP64 bit-exact, FP32 1e-6 (its bounds). Plane counts
around the 16 blocks (fewer planes than blocks, one each, a last block with fewer, several),
more columns than threads, one column per row. The larger volumes do not fit the cluster and
take the launch per half-sweep, with 2 and with more planes per thread."""
import numpy as np
import pytest

from conftest import rel
from test_gpu_rb_march import _sweeps

pytestmark = pytest.mark.gpu

SHAPES = [(5, 9, 12), (16, 8, 10), (17, 12, 9), (31, 5, 40), (33, 40, 7), (48, 44, 40), (64, 20, 64), (20, 140, 30),
          (90, 70, 66), (150, 90, 80)]


@pytest.mark.parametrize("bc_type, bc", [("dir", 0.3), ("neu", 0.0)])
@pytest.mark.parametrize("h", [(1.0, 1.0, 1.0), (0.7, 1.0, 1.5)])
@pytest.mark.parametrize("shape", SHAPES)
def test_cluster_sweeps(pkg, ctx, shape, h, bc_type, bc):
    rng = np.random.default_rng(shape[0] + 3 * shape[1])
    u = rng.standard_normal(shape)
    b = rng.standard_normal(shape)
    neu = bc_type == "neu"
    kw = dict(dt=0.8, bc=bc, bc_type=pkg.BC_NEU if neu else pkg.BC_DIR, tol=1e-30, max_sweeps=7, check_every=3, h=h)
    want = _sweeps(u, b, h, 0.8, bc, neu, 7)
    got = u.copy()
    ctx.poisson_solve(got, b, **kw)
    assert np.array_equal(got, want)
    got32 = u.astype(np.float32)
    ctx.poisson_solve(got32, b.astype(np.float32), **kw)
    assert rel(got32, want) <= 1e-6
