"""Timed cases of the framework's public entry points.

Kinds (the ``kind`` of a case):

* ``segment``   Context.rsfe_apply: a whole segmentation of one device-resident volume
                (the level set, the last solve's u and the fitting means), either in the
                production form (``solve``: red-black Gauss-Seidel to a relative residual
                of 1e-6) or in the reference constructor's form (``lex``: ls_steps
                lexicographic sweeps per outer iteration).
* ``batch``     Context.rsfe_apply_batched: uneven volumes through the stream queue.
* ``gauss``     Context.gauss_filter.
* ``poisson``   Context.poisson_solve.
* ``component`` Context.connected_component of a thresholded volume.
* ``conv``      Context.conv3d_bf16: one 3x3x3 convolution on the tensor cores.
* ``forward``   UNet.forward: the warm start's network.
* ``train``     UNet.train_step: one Adam step, with its gradients.

Volumes follow bench.py's workloads: ellipsoids on a noisy background under a linear
bias, the signed distance to a centred sphere as the initial level set. ``exact`` gives
the same results in 64 bits with plain torch.
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("3dimagetoolkit_b200")

DEV = "cuda" if torch.cuda.is_available() else "cpu"
_CTX = None


def context():
    """The program's one Context (a program keeps it for all its volumes)."""
    global _CTX
    if _CTX is None:
        _CTX = pkg.Context(0)
    return _CTX


# ------------------------------------------------------------------------ the cases
def _segment(name, nx, ny, nz, mode="solve", dtype="f32", bc="dir", sigma=3.0, hz=1.0, lamda2=1.0, maxiter=10):
    return {"name": name, "kind": "segment", "nx": nx, "ny": ny, "nz": nz, "mode": mode, "dtype": dtype,
            "bc": bc, "sigma": sigma, "hz": hz, "lamda2": lamda2, "maxiter": maxiter}


def listed():
    return [
        _segment("segment_48x44x40", 48, 44, 40, maxiter=5),
        _segment("segment_256", 256, 256, 256, maxiter=10),
        _segment("segment_512x512x320", 512, 512, 320, sigma=4.0, maxiter=5),
        _segment("segment_odd_neumann", 171, 203, 117, bc="neu", hz=1.5, lamda2=1.2, maxiter=10),
        _segment("segment_reference_f64", 64, 64, 64, mode="lex", dtype="f64", maxiter=5),
        {"name": "batch_8", "kind": "batch", "count": 8, "shapes_seed": 0, "maxiter": 5},
        {"name": "gauss_odd", "kind": "gauss", "nx": 225, "ny": 171, "nz": 203, "dtype": "f32", "sigma": 2.0,
         "hz": 1.5},
        {"name": "poisson_f64", "kind": "poisson", "nx": 128, "ny": 128, "nz": 128, "dtype": "f64", "bc": "dir"},
        {"name": "component_256", "kind": "component", "nx": 256, "ny": 256, "nz": 192, "dtype": "f32"},
        {"name": "conv_64", "kind": "conv", "cin": 32, "cout": 64, "nsamp": 1, "nx": 64, "ny": 64, "nz": 64},
        {"name": "unet_forward_128", "kind": "forward", "nsamp": 1, "nx": 128, "ny": 128, "nz": 128},
        {"name": "unet_train_128", "kind": "train", "nsamp": 1, "nx": 128, "ny": 128, "nz": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["segment"] * 5 + ["batch", "gauss", "poisson", "component", "conv", "forward", "train"])
    if kind == "segment":
        if rng.random() < 0.25:
            n = [_log_int(rng, 20, 72) for _ in range(3)]
            return {k: v for k, v in _segment("", *n, mode="lex", dtype=rng.choice(["f32", "f64"]),
                                              bc=rng.choice(["dir", "neu"]), maxiter=rng.randint(3, 6)).items()
                    if k != "name"}
        dtype = rng.choice(["f32", "f32", "f32", "f64"])
        n = [_log_int(rng, 36, 320 if dtype == "f32" else 200) for _ in range(3)]
        return {k: v for k, v in _segment("", *n, dtype=dtype,
                                          bc=rng.choice(["dir", "dir", "neu"]), sigma=rng.choice([2.0, 3.0, 3.0, 4.0]),
                                          hz=rng.choice([1.0, 1.0, 1.5]), lamda2=rng.choice([1.0, 1.0, 1.2]),
                                          maxiter=rng.randint(3, 6)).items() if k != "name"}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(4, 10), "shapes_seed": rng.randint(1, 10000),
                "maxiter": rng.randint(3, 5)}
    if kind == "gauss":
        return {"kind": "gauss", "nx": _log_int(rng, 24, 320), "ny": _log_int(rng, 24, 320),
                "nz": _log_int(rng, 24, 320), "dtype": rng.choice(["f32", "f32", "f64"]),
                "sigma": rng.choice([1.0, 2.0, 3.0, 4.0]), "hz": rng.choice([1.0, 1.5])}
    if kind == "poisson":
        return {"kind": "poisson", "nx": _log_int(rng, 24, 256), "ny": _log_int(rng, 24, 256),
                "nz": _log_int(rng, 24, 256), "dtype": rng.choice(["f32", "f64"]), "bc": rng.choice(["dir", "neu"])}
    if kind == "component":
        return {"kind": "component", "nx": _log_int(rng, 40, 320), "ny": _log_int(rng, 40, 320),
                "nz": _log_int(rng, 40, 320), "dtype": rng.choice(["f32", "f64"])}
    if kind == "conv":
        return {"kind": "conv", "cin": rng.choice([16, 32, 64]), "cout": rng.choice([16, 32, 64]),
                "nsamp": rng.randint(1, 2), "nx": _log_int(rng, 5, 96), "ny": _log_int(rng, 5, 96),
                "nz": rng.choice([16, 32, 48, 64, 96, 128])}
    nz = rng.choice([64, 128, 128, 256])
    return {"kind": kind, "nsamp": rng.randint(1, 2), "nx": 4 * _log_int(rng, 4, 32), "ny": 4 * _log_int(rng, 4, 32),
            "nz": nz}


# ----------------------------------------------------------------------- the inputs
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _dtype(case):
    return torch.float64 if case.get("dtype") == "f64" else torch.float32


def _grid(shape):
    return [torch.arange(n, dtype=torch.float64, device=DEV).reshape([-1 if a == q else 1 for q in range(3)])
            for a, n in enumerate(shape)]


def _ellipsoids(shape, seed, n, lo, hi, noise=0.05, salt=0):
    """Background 0.2, n ellipsoids of intensities 0.6-0.9, a bias 0.8-1.2 along k, noise."""
    rng = np.random.default_rng([int(seed), salt])
    g = _gen(seed, salt)
    gi, gj, gk = _grid(shape)
    dims = np.array(shape, dtype=np.float64)
    vol = torch.full(shape, 0.2, dtype=torch.float32, device=DEV)
    for _ in range(n):
        semi = np.minimum(rng.uniform(lo, hi, 3), (dims - 1) / 2.0)
        c = rng.uniform(semi, dims - 1 - semi)
        inside = ((gi - c[0]) / semi[0]) ** 2 + ((gj - c[1]) / semi[1]) ** 2 + ((gk - c[2]) / semi[2]) ** 2 <= 1.0
        vol[inside] = float(rng.uniform(0.6, 0.9))
    vol *= (0.8 + 0.4 * gk / max(shape[2] - 1, 1)).float()
    vol += noise * torch.randn(shape, generator=g, device=DEV)
    return vol


def _sphere(shape, radius):
    gi, gj, gk = _grid(shape)
    c = [(n - 1) / 2.0 for n in shape]
    return radius - torch.sqrt((gi - c[0]) ** 2 + (gj - c[1]) ** 2 + (gk - c[2]) ** 2)


def _shape(case):
    return (int(case["nx"]), int(case["ny"]), int(case["nz"]))


def _segment_inputs(case, seed):
    shape = _shape(case)
    u0 = _ellipsoids(shape, seed, 8, 0.08 * min(shape), 0.25 * min(shape))
    phi0 = _sphere(shape, 0.3 * min(shape))
    return u0.to(_dtype(case)).contiguous(), phi0.to(_dtype(case)).contiguous()


def _batch_inputs(case, seed):
    rng = np.random.default_rng(case["shapes_seed"])
    shapes = [(int(rng.integers(96, 257)), int(rng.integers(96, 257)), int(rng.integers(64, 193)))
              for _ in range(case["count"])]
    vols = [_ellipsoids(s, seed, 2, 8, 16, salt=q + 1) for q, s in enumerate(shapes)]
    return vols, [_sphere(s, 20.0).float() for s in shapes]


def _fields(case, seed):
    """The network's input fields as a segmentation meets them: a small forcing term, the
    previous u, div(d - b) and phi."""
    ns, shape = int(case["nsamp"]), _shape(case)
    x = torch.empty((ns, 4) + shape, dtype=torch.float32, device=DEV)
    for s in range(ns):
        g = _gen(seed, 77 + s)
        u0 = _ellipsoids(shape, seed, 3, 2, 2 + 0.3 * min(shape), salt=50 + s)
        phi = (u0 - 0.2).clamp(0, 1)
        x[s, 0] = 0.1 * (u0 - 0.5)
        x[s, 1] = phi + 0.02 * torch.randn(shape, generator=g, device=DEV)
        x[s, 2] = 0.05 * torch.randn(shape, generator=g, device=DEV)
        x[s, 3] = phi
    return x


# layers of the network in the order of its flat parameters
_CIN = [16, 16, 16, 32, 32, 64, 64, 32, 32, 16]
_COUT = [16, 16, 32, 32, 64, 64, 32, 32, 16, 16]


def _weights(seed):
    """Flat FP32 parameters: He-normal filters, small biases, a non-zero output layer."""
    rng = np.random.default_rng([int(seed), 4])
    parts = []
    for q, (ci, co) in enumerate(zip(_CIN, _COUT)):
        used = 4 if q == 0 else ci
        w = rng.standard_normal((co, ci, 27)) * math.sqrt(2.0 / (27 * used))
        w[:, used:] = 0
        parts += [w.ravel(), 0.05 * rng.standard_normal(co)]
    parts += [rng.standard_normal(8 * 64 * 32) * math.sqrt(2.0 / 64), 0.05 * rng.standard_normal(32)]
    parts += [rng.standard_normal(8 * 32 * 16) * math.sqrt(2.0 / 32), 0.05 * rng.standard_normal(16)]
    parts += [0.3 * rng.standard_normal(16), 0.05 * rng.standard_normal(1)]
    return np.concatenate(parts).astype(np.float32)


def _target(case, seed):
    shape = (int(case["nsamp"]),) + _shape(case)
    return 0.1 * torch.randn(shape, generator=_gen(seed, 91), device=DEV)


def _conv_inputs(case, seed):
    g = _gen(seed, 5)
    x = torch.randn((int(case["nsamp"]),) + _shape(case) + (int(case["cin"]),), generator=g, device=DEV).bfloat16()
    w = torch.randn((int(case["cout"]), int(case["cin"]), 3, 3, 3), generator=g, device=DEV)
    w = (w * math.sqrt(2.0 / (27 * case["cin"]))).bfloat16().float()
    return x, w, 0.1 * torch.randn(int(case["cout"]), generator=g, device=DEV)


def _poisson_inputs(case, seed):
    g = _gen(seed, 6)
    u = torch.rand(_shape(case), generator=g, device=DEV, dtype=_dtype(case))
    b = torch.rand(_shape(case), generator=g, device=DEV, dtype=_dtype(case)) - 0.5
    return u, b


def _component_input(case, seed):
    return _ellipsoids(_shape(case), seed, 8, 0.08 * min(_shape(case)), 0.3 * min(_shape(case)), noise=0.02).to(
        _dtype(case))


def _brightest(img):
    q = int(torch.argmax(img))
    n = img.shape
    return (q // (n[1] * n[2]), q // n[2] % n[1], q % n[2])


def _params(case):
    kw = dict(sigma=case.get("sigma", 3.0), lamda1=1.0, lamda2=case.get("lamda2", 1.0), epsilon=1e-3, lamda=0.5,
              maxiter=case["maxiter"], tol=0.0)
    if case.get("mode") == "lex":
        kw.update(ls_steps=5, sweep=pkg.SWEEP_LEXICOGRAPHIC)
    else:
        kw.update(ls_steps=1, gs_rel_res_tol=1e-6)
    kw["bc"] = pkg.BC_NEU if case.get("bc") == "neu" else pkg.BC_DIR
    return kw


def _h(case):
    return (1.0, 1.0, float(case.get("hz", 1.0)))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "segment":
        s["u0"], s["phi0"] = _segment_inputs(case, seed)
        s["params"] = pkg.default_params(**_params(case))
    elif kind == "batch":
        s["vols"], s["phi0"] = _batch_inputs(case, seed)
        s["params"] = pkg.default_params(**_params(case))
    elif kind == "gauss":
        s["x"] = _ellipsoids(_shape(case), seed, 8, 4, 40).to(_dtype(case))
    elif kind == "poisson":
        s["u"], s["b"] = _poisson_inputs(case, seed)
    elif kind == "component":
        s["x"] = _component_input(case, seed)
        s["ijk"] = _brightest(s["x"])
    elif kind == "conv":
        s["x"], s["w"], s["bias"] = _conv_inputs(case, seed)
    else:
        s["x"] = _fields(case, seed)
        if kind == "train":
            s["target"] = _target(case, seed)
        s["net"] = pkg.UNet(context(), seed=0)
        s["net"].set_params(_weights(seed))
    context()
    return s


def run(s):
    ctx, kind, case = context(), s["kind"], s["case"]
    if kind == "segment":
        r = ctx.rsfe_apply(s["u0"], s["phi0"], s["params"], h=_h(case), want_u=True, want_f=True)
        return {k: r[k] for k in ("phi", "u", "f1", "f2")}
    if kind == "batch":
        return ctx.rsfe_apply_batched(s["vols"], s["phi0"], s["params"])[0]
    if kind == "gauss":
        return ctx.gauss_filter(s["x"], case["sigma"], h=_h(case))
    if kind == "poisson":
        u = s["u"].clone()
        torch.cuda.current_stream().synchronize()  # the solve runs on the Context's own stream
        sweeps, rel, ok = ctx.poisson_solve(u, s["b"], bc_type=pkg.BC_NEU if case["bc"] == "neu" else pkg.BC_DIR)
        return {"u": u, "sweeps": sweeps, "converged": ok}
    if kind == "component":
        return ctx.connected_component(s["x"], ijk=s["ijk"])
    if kind == "conv":
        return ctx.conv3d_bf16(s["x"], s["w"], s["bias"])
    if kind == "forward":
        return s["net"].forward(s["x"])
    loss, grads = s["net"].train_step(s["x"], s["target"], 1e-3, want_grads=True)
    return {"loss": loss, "grads": grads}


# -------------------------------------------------------------------------- the work
def _taps(sigma, h):
    n = math.ceil(2 * 3.0 * sigma / h)
    return n if n % 2 else n + 1


def _voxels(case):
    return int(case["nx"]) * int(case["ny"]) * int(case["nz"])


def _solve_work(n, es, sweeps):
    """u read and written, b read per sweep; 10 operations a cell."""
    return 3 * n * es * sweeps, 10.0 * n * sweeps


def _segment_work(n, es, case):
    """One outer iteration reads u0, g, phi and the three b and writes phi and b, and its
    sweeps (about 35 to the residual) read u and b and write u; the four fields' and the
    pair's convolutions are 2 taps operations per field and axis."""
    taps = _taps(case.get("sigma", 3.0), 1.0)
    sweeps = 5 if case.get("mode") == "lex" else 35
    sb, sf = _solve_work(n, es, sweeps)
    by = case["maxiter"] * (n * es * (3 + 3 + 4) + sb) + 4 * n * es
    return by, case["maxiter"] * (n * (6 * 3 * 2 * taps + 60.0) + sf)


def work(case):
    kind = case["kind"]
    es = 8 if case.get("dtype") == "f64" else 4
    if kind == "segment":
        by, fl = _segment_work(_voxels(case), es, case)
    elif kind == "batch":
        rng = np.random.default_rng(case["shapes_seed"])
        n = sum(int(rng.integers(96, 257)) * int(rng.integers(96, 257)) * int(rng.integers(64, 193))
                for _ in range(case["count"]))
        by, fl = _segment_work(n, 4, case)
    elif kind == "gauss":
        by, fl = 2 * es * _voxels(case), 2.0 * _voxels(case) * (2 * _taps(case["sigma"], 1.0) +
                                                                _taps(case["sigma"], case["hz"]))
    elif kind == "poisson":
        by, fl = _solve_work(_voxels(case), es, 35)
    elif kind == "component":
        by, fl = 2 * es * _voxels(case), 0.0
    elif kind == "conv":
        n = case["nsamp"] * _voxels(case)
        by = n * (2 * case["cin"] + 4 * case["cout"])
        fl = 2.0 * 27 * n * case["cin"] * case["cout"]
    else:
        n = case["nsamp"] * _voxels(case)
        scale = [1, 1, 8, 8, 64, 64, 8, 8, 1, 1]
        cin = [4] + _CIN[1:]
        fl = sum(2.0 * 27 * n / q * ci * co for q, ci, co in zip(scale, cin, _COUT))
        fl += 2.0 * n * (64 * 32 / 8 + 32 * 16 + 16)
        by = n * 4 * 5
        if kind == "train":
            fl, by = 3 * fl, n * 4 * 5 + 4 * len(_weights(0)) * 5
    return {"bytes": float(by), "flops": float(fl)}


# ------------------------------------------------------- the same results in 64 bits
def _at(x, axis, lo, hi):
    return x.narrow(axis, lo, hi - lo)


def _conv_axis(x, axis, sigma, h):
    """Normalised Gaussian along one axis, zero outside."""
    n = _taps(sigma, h)
    S = n // 2
    t = np.arange(n) - S
    w = np.exp(-t * t * h * h / (2 * sigma * sigma))
    w /= w.sum()
    L = x.shape[axis]
    out = torch.zeros_like(x)
    for q in range(n):
        o = q - S
        lo, hi = max(0, -o), min(L, L - o)
        if lo < hi:
            _at(out, axis, lo, hi).add_(_at(x, axis, lo + o, hi + o), alpha=float(w[q]))
    return out


def _gauss(x, sigma, h):
    for a in (2, 1, 0):
        x = _conv_axis(x, a, sigma, h[a])
    return x


def _grad_axis(f, axis, h):
    L = f.shape[axis]
    g = torch.empty_like(f)
    _at(g, axis, 1, L - 1).copy_((_at(f, axis, 2, L) - _at(f, axis, 0, L - 2)) / (2 * h))
    _at(g, axis, 0, 1).copy_((4 * _at(f, axis, 1, 2) - 3 * _at(f, axis, 0, 1) - _at(f, axis, 2, 3)) / (2 * h))
    _at(g, axis, L - 1, L).copy_((3 * _at(f, axis, L - 1, L) - 4 * _at(f, axis, L - 2, L - 1) +
                                  _at(f, axis, L - 3, L - 2)) / (2 * h))
    return g


def _div(v, h):
    """Divergence by the same differences, with the two face and edge rules of image3d's div."""
    tx, tz = _grad_axis(v[0], 0, h[0]), _grad_axis(v[2], 2, h[2])
    X = v[0]
    tx[-1, 1:-1, 1:-1] = ((3 * X[-1] - 4 * X[-2] + X[-3]) / 2 * h[0])[1:-1, 1:-1]
    Z = v[2]
    tz[1:-1, 0, -1] = ((3 * Z[:, 0, -1] - 4 * Z[:, 0, -2] + Z[:, 0, -2]) / (2 * h[2]))[1:-1]
    return tx + _grad_axis(v[1], 1, h[1]) + tz


def _neighbours(u, h):
    """Sum of the six neighbours over h^2, nothing from outside."""
    s = torch.zeros_like(u)
    for a in range(3):
        L, w = u.shape[a], 1.0 / (h[a] * h[a])
        _at(s, a, 0, L - 1).add_(_at(u, a, 1, L), alpha=w)
        _at(s, a, 1, L).add_(_at(u, a, 0, L - 1), alpha=w)
    return s


def _diagonal(shape, h, dt, neu):
    d = torch.full(shape, 1.0 / dt, dtype=torch.float64, device=DEV)
    for a in range(3):
        c = torch.full((shape[a],), 2.0, dtype=torch.float64, device=DEV)
        if neu:
            c[0] = c[-1] = 1.0
        d += (c / (h[a] * h[a])).reshape([-1 if q == a else 1 for q in range(3)])
    return d


def _unknowns(shape, neu):
    m = torch.ones(shape, dtype=torch.bool, device=DEV)
    if not neu:
        for a in range(3):
            _at(m, a, 0, 1).fill_(False)
            _at(m, a, shape[a] - 1, shape[a]).fill_(False)
    return m


def _faces(u, value):
    for a in range(3):
        _at(u, a, 0, 1).fill_(value)
        _at(u, a, u.shape[a] - 1, u.shape[a]).fill_(value)


def _solve(u, b, h, dt, neu, tol, first, rate0):
    """Red-black Gauss-Seidel for (1/dt - Laplace) u = b to a relative residual, checked when
    the contraction rate says that it is reached. Returns sweeps and the rate."""
    shape = tuple(u.shape)
    diag, live = _diagonal(shape, h, dt, neu), _unknowns(shape, neu)
    gi, gj, gk = [torch.arange(n, device=DEV).reshape([-1 if a == q else 1 for q in range(3)])
                  for a, n in enumerate(shape)]
    red = ((gi + gj + gk) % 2 == 0)
    masks = [live & red, live & ~red]
    norm = math.sqrt(float((b * b * live).sum()))
    s, s_prev, r_prev, used = 0, 0, -1.0, 0.0
    nxt = first if first > 0 else 4
    while s < 1000:
        for m in masks:
            torch.where(m, (_neighbours(u, h) + b) / diag, u, out=u)
        s += 1
        if s < nxt and s < 1000:
            continue
        res = (_neighbours(u, h) + b - diag * u) * live
        r = math.sqrt(float((res * res).sum()))
        r = r / norm if norm > 0 else r
        if r <= tol:
            break
        if s_prev > 0 and r_prev > r > 0:
            rate = (r / r_prev) ** (1.0 / (s - s_prev))
        elif 0 < rate0 < 1 and r > 0:
            rate = rate0
        else:
            rate = 0.0
        step = 4
        if rate:
            used = rate
            need = math.log(tol / r) / math.log(rate)
            step = max(1, int(math.ceil(need)) if need < 32 else 32)
        nxt, s_prev, r_prev = min(1000, s + step), s, r
    return s, (used if used > 0 else rate0)


def _lex(u, b, h, dt, neu, sweeps):
    """Lexicographic Gauss-Seidel sweeps, one plane i + j + k = s after another."""
    shape = tuple(u.shape)
    if not neu:
        _faces(u, 0.0)
    diag = _diagonal(shape, h, dt, neu)
    p = [n + 2 for n in shape]
    up = torch.zeros(p, dtype=torch.float64, device=DEV)
    up[1:-1, 1:-1, 1:-1] = u
    st = (p[1] * p[2], p[2], 1)
    gi, gj, gk = torch.meshgrid(*[torch.arange(n, device=DEV) for n in shape], indexing="ij")
    live = _unknowns(shape, neu)
    plane = (gi + gj + gk)[live]
    own = (gi * (shape[1] * shape[2]) + gj * shape[2] + gk)[live]
    pad = ((gi + 1) * st[0] + (gj + 1) * st[1] + gk + 1)[live]
    order = torch.argsort(plane, stable=True)
    counts = torch.bincount(plane).tolist()
    own, pad = own[order].split(counts), pad[order].split(counts)
    uf, bf, df = up.view(-1), b.reshape(-1), diag.reshape(-1)
    for _ in range(sweeps):
        for q, c in enumerate(counts):
            if not c:
                continue
            o, f = own[q], pad[q]
            acc = bf[o] + uf[f] / dt
            for a in range(3):
                acc = acc + (uf[f - st[a]] + uf[f + st[a]]) / (h[a] * h[a])
            uf[f] = acc / df[o]
    u.copy_(up[1:-1, 1:-1, 1:-1])


def _shrink(x, g):
    return torch.sign(x) * (x.abs() - g).clamp_min(0)


def _exact_segment(case, u0, phi0):
    u0, phi, h = u0.double(), phi0.double(), _h(case)
    sigma, l1, l2, lam, dt = case.get("sigma", 3.0), 1.0, case.get("lamda2", 1.0), 0.5, 1.0
    neu = case.get("bc") == "neu"
    phi = (phi - phi.min()) / (phi.max() - phi.min())
    kones = _gauss(torch.ones_like(u0), sigma, h) if l1 != l2 else None
    g = 1.0 / (lam * (1 + 100.0 * sum(_grad_axis(u0, a, h[a]) ** 2 for a in range(3))))
    b = [torch.zeros_like(u0) for _ in range(3)]
    divdb = torch.zeros_like(u0)
    first, rate = 0, 0.0
    for _ in range(case["maxiter"]):
        H = torch.atan((phi - 0.5) / 1e-3) / math.pi
        H, Hb = 0.5 + H, 0.5 - H
        f1 = _gauss(H * u0, sigma, h) / _gauss(H, sigma, h)
        f2 = _gauss(Hb * u0, sigma, h) / _gauss(Hb, sigma, h)
        del H, Hb
        rhs = 2 * u0 * _gauss(l1 * f1 - l2 * f2, sigma, h) - _gauss(l1 * f1 * f1 - l2 * f2 * f2, sigma, h)
        if kones is not None:
            rhs -= (l1 - l2) * u0 * u0 * kones
        rhs = rhs / lam - divdb
        old, u = phi, phi.clone()
        if case.get("mode") == "lex":
            _lex(u, rhs, h, dt, neu, 5)
        else:
            if not neu:
                _faces(u, 0.0)
            first, rate = _solve(u, rhs + u / dt, h, dt, neu, 1e-6, first, rate)
        phi = u.clamp(0, 1)
        d = []
        for a in range(3):
            s = b[a] + _grad_axis(phi, a, h[a])
            t = _shrink(s, g)
            b[a] = s - t
            d.append(t - b[a])
        divdb = _div(d, h)
        del old, d
    return {"phi": phi, "u": u, "f1": f1, "f2": f2}


def _exact_component(img, ijk):
    shape = tuple(img.shape)
    I, J, K = (min(max(c, 1), n - 2) for c, n in zip(ijk, shape))
    mn, mx = img.min(), img.max()
    pivot = (mn.double() + (mx - mn).double() * 0.5).to(img.dtype)
    white = img < pivot if bool(img[I, J, K] < pivot) else img >= pivot
    spread = _unknowns(shape, False)
    m = torch.zeros(shape, dtype=torch.bool, device=DEV)
    m[I, J, K] = True
    count = 1
    while True:
        for _ in range(16):
            s = m & spread
            for a in range(3):
                L = shape[a]
                _at(m, a, 0, L - 1).logical_or_(_at(s, a, 1, L))
                _at(m, a, 1, L).logical_or_(_at(s, a, 0, L - 1))
            m &= white
        m[I, J, K] = True
        now = int(m.sum())
        if now == count:
            return m.double()
        count = now


def _unflatten(flat):
    ps, o = [], 0
    for ci, co in zip(_CIN, _COUT):
        w = flat[o:o + co * ci * 27].reshape(co, ci, 3, 3, 3)
        o += co * ci * 27
        ps.append((w, flat[o:o + co]))
        o += co
    ups = []
    for ci, co in ((64, 32), (32, 16)):
        # U[8][cin][cout], child 4 di + 2 dj + dk -> conv_transpose3d's [cin][cout][2][2][2]
        w = flat[o:o + 8 * ci * co].reshape(2, 2, 2, ci, co).permute(3, 4, 0, 1, 2)
        o += 8 * ci * co
        ups.append((w, flat[o:o + co]))
        o += co
    return ps, ups, flat[o:o + 16], flat[o + 16]


def _exact_net(x, flat):
    F = torch.nn.functional
    ps, ups, ow, ob = _unflatten(flat)

    def c(q, v):
        return F.relu(F.conv3d(v, ps[q][0], ps[q][1], padding=1))

    v = torch.cat([x, torch.zeros((x.shape[0], 12) + tuple(x.shape[2:]), dtype=x.dtype, device=x.device)], 1)
    a = c(1, c(0, v))
    b = c(3, c(2, F.max_pool3d(a, 2)))
    e = c(5, c(4, F.max_pool3d(b, 2)))
    d2 = c(7, c(6, torch.cat([F.conv_transpose3d(e, ups[0][0], ups[0][1], stride=2), b], 1)))
    d1 = c(9, c(8, torch.cat([F.conv_transpose3d(d2, ups[1][0], ups[1][1], stride=2), a], 1)))
    return (d1 * ow.reshape(1, -1, 1, 1, 1)).sum(1) + ob


def exact(case, seed):
    kind = case["kind"]
    if kind == "segment":
        return _exact_segment(case, *_segment_inputs(case, seed))
    if kind == "batch":
        return [_exact_segment(case, v, p)["phi"] for v, p in zip(*_batch_inputs(case, seed))]
    if kind == "gauss":
        x = _ellipsoids(_shape(case), seed, 8, 4, 40).to(_dtype(case)).double()
        return _gauss(x, case["sigma"], _h(case))
    if kind == "poisson":
        u, b = (v.double() for v in _poisson_inputs(case, seed))
        neu = case["bc"] == "neu"
        if not neu:
            _faces(u, 0.0)
        _solve(u, b + u, (1.0, 1.0, 1.0), 1.0, neu, 1e-6, 0, 0.0)
        return {"u": u, "sweeps": None, "converged": None}
    if kind == "component":
        x = _component_input(case, seed)
        return _exact_component(x, _brightest(x))
    if kind == "conv":
        x, w, b = _conv_inputs(case, seed)
        y = torch.nn.functional.conv3d(x.double().permute(0, 4, 1, 2, 3), w.double(), b.double(), padding=1)
        return y.permute(0, 2, 3, 4, 1).contiguous()
    x, flat = _fields(case, seed).double(), torch.tensor(_weights(seed), dtype=torch.float64, device=DEV)
    if kind == "forward":
        return _exact_net(x, flat)
    flat.requires_grad_(True)
    loss = ((_exact_net(x, flat) - _target(case, seed).double()) ** 2).mean()
    loss.backward()
    return {"loss": float(loss), "grads": flat.grad}
