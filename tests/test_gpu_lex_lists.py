"""GPU: the task list of the lexicographic sweeps (lex_tile_kernel), which the context keeps from
call to call. Sweeps in FP64 are bit-exact against the oracle's sequential loops."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _case(shape, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(shape), rng.standard_normal(shape)


def _sweep(c, u, b, sweeps, **kw):
    """The sweeps on device arrays (the context then needs no buffers of its own for them)."""
    du, db = torch.from_numpy(u.copy()).cuda(), torch.from_numpy(b).cuda()
    torch.cuda.synchronize()
    c.poisson_sweeps(du, db, sweeps=sweeps, **kw)
    return du.cpu().numpy()


def test_list_after_a_failed_allocation(pkg, O):
    """A larger list that finds no device memory costs the context its old list: the next call of
    the old size must write its list again (it took whatever the new buffer held)."""
    u, b = _case((40, 37, 52), 3)
    want = O.poisson_sweeps(u, b, dt=1.0, bc=0.0, bc_type=pkg.BC_DIR, sweeps=3, h=(1.0, 1.0, 1.0))
    big = torch.zeros((258, 258, 258), device="cuda")
    with pkg.Context(0) as c:
        c.poisson_sweeps(big, big.clone(), sweeps=1)
        first = _sweep(c, u, b, 3)
        # 4096 tiles x 512 sweeps: a list of 16 MB, with 6 MB left on the device
        rhs = big.clone()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        hold = torch.empty(free - (6 << 20), dtype=torch.uint8, device="cuda")
        try:
            c.poisson_sweeps(big, rhs, sweeps=512)
        except pkg.Im3dError as e:
            assert e.status == 5  # out of memory
        del hold
        torch.cuda.empty_cache()
        again = _sweep(c, u, b, 3)
    assert np.array_equal(first, want)
    assert np.array_equal(again, want)


@pytest.mark.parametrize("bc_type, bc", [("dir", 0.3), ("neu", 0.3)])
@pytest.mark.parametrize("limit", [1, 4000, 8 * 27 * 4 + 4 * 28 + 256 + 16])
def test_sweeps_under_a_memory_limit(pkg, O, limit, bc_type, bc):
    """On device arrays the sweeps need no memory: any limit lets them run, without the list, with
    a list of one sweep, or with the whole one; and the list gives way to a buffer that another
    call needs under the same limit."""
    u, b = _case((40, 37, 48), 5)  # 27 tiles (Dirichlet and Neumann)
    kw = dict(dt=0.7, bc=bc, bc_type=pkg.BC_NEU if bc_type == "neu" else pkg.BC_DIR, h=(0.8, 1.0, 1.3))
    want = O.poisson_sweeps(u, b, sweeps=4, **kw)
    with pkg.Context(0) as c:
        c.set_option(pkg.OPT_DEVICE_MEMORY_LIMIT, limit)
        got = _sweep(c, u, b, 4, **kw)
        assert np.array_equal(got, want)
        # two host arrays need two buffers of this size, and leave no room for the list
        c.set_option(pkg.OPT_DEVICE_MEMORY_LIMIT, 2 * (u.size * 8 + 256) + 1)
        got = u.copy()
        c.poisson_sweeps(got, b, sweeps=4, **kw)
        assert np.array_equal(got, want)
        c.set_option(pkg.OPT_DEVICE_MEMORY_LIMIT, 0)
        assert np.array_equal(_sweep(c, u, b, 4, **kw), want)


def test_rows_of_more_than_65536_tiles(pkg, ctx, O):
    """A tile's k index has more than 16 bits where nz is above 2^20 (3 x 3 x 1049000)."""
    u, b = _case((3, 3, 1049000), 7)
    kw = dict(dt=0.7, bc=0.0, bc_type=pkg.BC_DIR, sweeps=2, h=(1.0, 1.0, 1.0))
    want = O.poisson_sweeps(u, b, **kw)
    got = u.copy()
    ctx.poisson_sweeps(got, b, **kw)
    assert np.array_equal(got, want)


def test_sweeps_of_an_iteration_are_bounded(pkg, ctx):
    """At most 100000 sweeps per outer iteration, also where their number is known beforehand."""
    u0 = pkg.synth.ellipsoids((8, 8, 8), 3, n=1, semi_axes=(2, 3))
    phi0 = pkg.synth.sphere_phi0((8, 8, 8), 2.5)
    params = pkg.default_params(sigma=1.0, lamda1=1.0, lamda2=1.0, epsilon=1e-3, lamda=0.5, tol=0.0, maxiter=1,
                                ls_steps=100003, sweep=pkg.SWEEP_LEXICOGRAPHIC)
    stats = ctx.rsfe_apply(u0, phi0, params)["stats"]
    assert stats["total_sweeps"] == 100000 and stats["not_converged"] == 1
