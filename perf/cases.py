"""What a user of this framework runs, as measurable cases.

Every case is one call of the public interface that a run script makes over
and over: a timestep of one of the physics classes (``RK2mid`` / ``RK2trap`` /
``RK4`` ``.do_advance``), a right-hand side (``RHS``), the lazy switch of a
field between grid space and k-space, one step of an uneven ensemble, one step
of the closed LES, one training step of its network.  Grid sizes, viscosities
and time steps are those of the benchmark configurations and of the tests.

States are seeded random-phase solenoidal fields with a developed spectrum (a
k^4 rise, a k^(-5/3) range and a viscous cut), 2/3 dealiased, made on the GPU.
``exact`` advances the same inputs with plain torch transforms and arithmetic
in 64 bits.
"""
import math
import os

import numpy as np
import torch

from __graft_entry__ import load_package

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_LEN = [16, 24, 32, 48, 64, 96, 128, 192, 256, 512]      # transform lengths in use


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest configured run: 2D turbulence, launch- and latency-bound
        dict(name="hydro2d_128", kind="step2d", physics="hydro", ny=128, nx=128, precision="fp64"),
        # one convection run of the ensemble's largest size by itself
        dict(name="bouss2d_512", kind="step2d", physics="bouss", ny=512, nx=512, precision="fp64"),
        # the headline: 3D turbulence in FP64
        dict(name="hydro3d_256", kind="step3d", physics="hydro", nz=256, ny=256, nx=256, precision="fp64"),
        # the same run with FP32 transforms
        dict(name="hydro3d_256_fp32", kind="step3d", physics="hydro", nz=256, ny=256, nx=256, precision="fp32"),
        # a medium MHD run in FP64
        dict(name="mhd3d_128", kind="step3d", physics="mhd", nz=128, ny=128, nx=128, precision="fp64"),
        # the configured MHD run with FP32 transforms
        dict(name="mhd3d_256_fp32", kind="step3d", physics="mhd", nz=256, ny=256, nx=256, precision="fp32"),
        # a right-hand side for a user's own integrator, on a box of three different sides (3 x 2^k too)
        dict(name="rhs3d_48x192x96", kind="rhs3d", physics="hydro", nz=48, ny=192, nx=96, precision="fp64"),
        # a vector field to grid space and back: output, analysis, setting of initial conditions
        dict(name="transform3d_192x128x256", kind="transform", nz=192, ny=128, nx=256),
        # convection in a rotating box: the reference's own sequence of operators, trapezoidal steps
        dict(name="rotbouss3d_64", kind="generic3d", nz=64, ny=64, nx=64),
        # a quarter of the configured ensemble of uneven 2D convection runs, one graph launch per step
        dict(name="ensemble_128runs", kind="ensemble", n64=33, n128=31, n256=29, n512=35, precision="fp64"),
        # the coarse LES with the learned closure
        dict(name="les3d_64", kind="les", n=64, precision="fp32"),
        # one optimiser step of the closure network: forward, backward, update
        dict(name="train_65536", kind="train", samples=65536),
    ]


def draw(rng):
    kind = rng.choice(["step2d", "step2d", "step3d", "step3d", "rhs3d", "transform", "generic3d", "ensemble", "les",
                       "train"])
    if kind == "step2d":
        sizes = [n for n in _LEN if n >= 32]
        return dict(kind=kind, physics=rng.choice(["hydro", "bouss"]), ny=rng.choice(sizes), nx=rng.choice(sizes),
                    precision=rng.choice(["fp64", "fp64", "fp32"]))
    if kind in ("step3d", "rhs3d"):
        physics, precision = rng.choice(["hydro", "hydro", "mhd"]), rng.choice(["fp64", "fp64", "fp32", "df64"])
        sizes = [16, 32, 64, 128, 256] if precision == "df64" else _LEN[:-1]
        most = 128 ** 3 * (2 if physics == "mhd" else 4) * (2 if precision != "fp64" else 1)
        return dict(kind=kind, physics="hydro" if precision == "df64" else physics, precision=precision,
                    **_box(rng, sizes, most))
    if kind == "transform":
        return dict(kind=kind, **_box(rng, _LEN, 256 ** 3))
    if kind == "generic3d":
        return dict(kind=kind, **_box(rng, _LEN[:-1], 96 ** 3))
    if kind == "ensemble":
        return dict(kind=kind, precision=rng.choice(["fp64", "fp32"]), n64=rng.randint(1, 48), n128=rng.randint(1, 48),
                    n256=rng.randint(1, 40), n512=rng.randint(1, 35))
    if kind == "les":
        return dict(kind=kind, n=rng.choice([32, 48, 64]), precision=rng.choice(["fp32", "fp64"]))
    return dict(kind=kind, samples=int(round(math.exp(rng.uniform(math.log(1000), math.log(200000))))))


def _box(rng, sizes, most):
    while True:
        nz, ny, nx = (rng.choice(sizes) for _ in range(3))
        if 16 ** 3 <= nz * ny * nx <= most:
            return dict(nz=nz, ny=ny, nx=nx)


# ------------------------------------------------------------------ inputs
def _shape(case):
    return tuple(case[n] for n in ("nz", "ny", "nx") if n in case)


def _kvec(shape, device="cuda"):
    """Wavenumbers of a 2 pi box in the k layout: (kx, ky, kz) over [ky][kz][kx] in 3D, (kx, ky) over [kx][ky] in 2D."""
    f = [torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=device) for n in shape]
    kx = torch.arange(shape[-1] // 2 + 1, dtype=torch.float64, device=device)
    if len(shape) == 3:
        return kx[None, None, :], f[1][:, None, None], f[0][None, :, None]
    return kx[:, None], f[0][None, :]


def _kept(shape):
    n = (shape[-1], shape[-2]) + tuple(shape[:1] if len(shape) == 3 else ())
    keep = True
    for k, m in zip(_kvec(shape), n):
        keep = keep & (k.abs() < m / 3.0)
    return keep


def _fwd(x):
    """The forward transform (1/N, k layout) of x[(z,) y, x]."""
    h = torch.fft.rfftn(x) / x.numel()
    return (h.permute(1, 0, 2) if x.dim() == 3 else h.permute(1, 0)).contiguous()


def _bwd(k, shape):
    h = k.permute(1, 0, 2) if k.dim() == 3 else k.permute(1, 0)
    return torch.fft.irfftn(h, s=shape) * math.prod(shape)


def _field(shape, gen, k0):
    """A random-phase scalar with a developed spectrum, dealiased."""
    ks = _kvec(shape)
    kk = torch.sqrt(sum(k * k for k in ks))
    kmax = min(shape) / 3.0
    energy = kk ** 4 * (1 + (kk / k0) ** 2) ** (-17.0 / 6.0) * torch.exp(-4.0 * kk / kmax)
    amp = torch.sqrt(energy) / torch.where(kk > 0, kk, torch.ones_like(kk)) ** ((len(shape) - 1) / 2.0)
    h = _fwd(torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen))
    return torch.where(_kept(shape), amp * h / torch.where(h == 0, torch.ones_like(h), h).abs(), torch.zeros_like(h))


def _mean_square(h):
    """<|f|^2> from the k array of f (the kx > 0 half counted twice)."""
    a = (h.real ** 2 + h.imag ** 2)
    first = a[..., 0] if h.dim() == 3 else a[0]
    return 2 * a.sum() - first.sum()


def _scalar(shape, gen, rms, k0=4.0):
    h = _field(shape, gen, k0)
    return h * (rms / torch.sqrt(_mean_square(h)))


def _vector(shape, gen, k0=4.0):
    """A solenoidal vector of unit energy 1/2 <|u|^2>."""
    ks = _kvec(shape)
    k2 = sum(k * k for k in ks)
    k2 = torch.where(k2 == 0, torch.ones_like(k2), k2)
    u = [_field(shape, gen, k0) for _ in ks]
    div = sum(k * c for k, c in zip(ks, u)) / k2
    u = [c - k * div for k, c in zip(ks, u)]
    s = math.sqrt(2.0 / float(sum(_mean_square(c) for c in u)))
    return [(c * s).contiguous() for c in u]


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _inputs(case, seed):
    """{field: [k arrays]} of a single run."""
    shape, gen = _shape(case), _gen(seed)
    out = {"u": _vector(shape, gen, 3.0 if case.get("physics") == "mhd" else 4.0)}
    if case.get("physics") == "mhd":
        out["B"] = _vector(shape, gen, 3.0)
    if case.get("physics") == "bouss" or case["kind"] == "generic3d":
        out["T"] = [_scalar(shape, gen, 0.1)]
    return out


_CLASSES = [64, 128, 256, 512]


def _ensemble_inputs(case, seed):
    """Per size class a slab [run][u_x, u_y, T][kx][ky]."""
    out = []
    for n in _CLASSES:
        gen = _gen(seed, n)
        runs = [torch.stack(_vector((n, n), gen) + [_scalar((n, n), gen, 0.1)]) for _ in range(case["n%d" % n])]
        out.append(torch.stack(runs))
    return out


def _train_inputs(case, seed):
    """Normalised gradient inputs [n][16] (10 used), targets [n][8] (6 used) and starting parameters."""
    n, gen = case["samples"], _gen(seed)
    g = torch.randn((n, 9), generator=gen, device="cuda") * (1 + torch.rand((n, 1), generator=gen, device="cuda"))
    X = torch.zeros((n, 16), device="cuda")
    X[:, :9], X[:, 9] = g, 1.0
    T = torch.zeros((n, 8), device="cuda")
    T[:, :6] = 0.3 * g[:, :6] * g[:, 3:9] + torch.randn((n, 6), generator=gen, device="cuda")
    p = []
    for fo, fi, rows, cols in ((64, 16, 64, 10), (64, 64, 64, 64), (8, 64, 6, 64)):
        w = torch.zeros((fo, fi), device="cuda")
        w[:rows, :cols] = (torch.rand((rows, cols), generator=gen, device="cuda") * 2 - 1) * math.sqrt(6.0 / (rows + cols))
        p += [w.reshape(-1), torch.zeros(fo, device="cuda")]
    return X.to(torch.bfloat16), T, torch.cat(p)


# ------------------------------------------------------------------ programs
_DT = {"hydro": 2e-3, "mhd": 1e-3, "bouss": 1e-2}
_OMEGA = (0.5, -0.2, 0.3)                                     # (z, y, x), the grid's axis order


def _physics(dd, case):
    M, shape = dd.mods, _shape(case)
    if case["kind"] == "generic3d":
        rhs = M.BoussinesqHydro(shape, M.FourierRepresentation)
        rhs.parameters.update(nu=5e-3, kappa=5e-3, Omega=np.array(_OMEGA), boussinesq_direction="z")
        return rhs
    rhs = {"hydro": M.IncompressibleHydro, "mhd": M.IncompressibleMHD, "bouss": M.BoussinesqHydro}[case["physics"]](
        shape, M.FourierRepresentation)
    if case["physics"] == "bouss":
        rhs.parameters.update(nu=2e-3, kappa=2e-3, boussinesq_direction="y")
    elif case["physics"] == "mhd":
        rhs.parameters.update(nu=5e-3, eta=5e-3)
    else:
        rhs.parameters.update(nu=1e-3 if len(shape) == 2 else 5e-3)
    return rhs


def _dt(case):
    if case["kind"] == "generic3d":
        return 2e-3
    return 1e-3 if case["kind"] == "step2d" and case["physics"] == "hydro" else _DT[case.get("physics", "hydro")]


def prepare(case, seed):
    dd = load_package()
    kind = case["kind"]
    s = dict(case=case, dd=dd)
    if kind == "ensemble":
        sizes = [n for n in _CLASSES for _ in range(case["n%d" % n])]
        ens = dd.ensemble.BoussinesqEnsemble2D(sizes, precision=case["precision"])
        r = 0
        for slab in _ensemble_inputs(case, seed):
            for run in slab.cpu().numpy():
                ens.set_run_state(r, run)
                r += 1
        s["ens"] = ens
        return s
    if kind == "train":
        X, T, p = _train_inputs(case, seed)
        net = dd.closure.MLPClosure(math.pi / 21.0)
        net.params.copy_(p)
        net.pack()
        s.update(X=X, T=T, net=net)
        return s
    M = dd.mods
    dd.config.decfg.set("FFT", "precision", case.get("precision", "fp64"))
    if kind == "les":
        case = dict(case, nz=case["n"], ny=case["n"], nx=case["n"], physics="hydro")
        rhs = M.LESHydro(_shape(case), M.FourierRepresentation, closure=dd.closure.MLPClosure.load(),
                         precision=case["precision"])
        rhs.parameters["nu"] = 5e-3
    elif kind == "transform":
        rhs = M.IncompressibleHydro(_shape(case), M.FourierRepresentation)
    else:
        rhs = _physics(dd, case)
    data = rhs.create_fields(0.0)
    for name, comps in _inputs(case, seed).items():
        for i, c in enumerate(comps):
            data[name][i]["kspace"] = c
    s.update(rhs=rhs, data=data, dt=_dt(case))
    if kind == "rhs3d":
        s["deriv"] = rhs.create_fields(0.0)
    elif kind == "step2d":
        s["ti"] = M.RK2mid(rhs)
    elif kind == "generic3d":
        s["ti"] = M.RK2trap(rhs)
    elif kind != "transform":
        s["ti"] = M.RK4(rhs)
    return s


def _kdata(data):
    return {name: [c.kdata for _, c in field] for name, field in data}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "ensemble":
        s["ens"].step(1e-2)
        return [c.slab for c in s["ens"].classes]
    if kind == "train":
        grad, loss = s["net"].gradient(s["X"], s["T"])
        s["net"].adam(1e-3)
        return dict(grad=grad, loss=loss, params=s["net"].params)
    s["dd"].config.decfg.set("FFT", "precision", case.get("precision", "fp64"))
    if kind == "transform":
        x = [c["xspace"] for _, c in s["data"]["u"]]
        k = [c["kspace"] for _, c in s["data"]["u"]]
        return dict(x=x, k=k)
    if kind == "rhs3d":
        s["rhs"].RHS(s["data"], s["deriv"])
        return _kdata(s["deriv"])
    s["ti"].do_advance(s["data"], s["dt"])
    return _kdata(s["data"])


# ------------------------------------------------------------------ work
def _transforms(n, count):
    """Flops of `count` real transforms of n points."""
    return count * 2.5 * n * math.log2(n)


def work(case):
    kind = case["kind"]
    if kind == "train":
        n, weights = case["samples"], 10 * 64 + 64 * 64 + 64 * 6
        return {"bytes": n * (32 + 32) + 5 * 4 * (weights + 134), "flops": 6.0 * n * weights}
    if kind == "ensemble":
        b = f = 0.0
        for n in _CLASSES:
            b += case["n%d" % n] * 2 * 3 * 16 * (n // 2 + 1) * n
            f += case["n%d" % n] * 2 * _transforms(n * n, 7)
        return {"bytes": b, "flops": f}
    shape = (case["n"],) * 3 if kind == "les" else _shape(case)
    n, kc = math.prod(shape), math.prod(shape[:-1]) * (shape[-1] // 2 + 1)
    d = len(shape)
    if kind == "transform":
        return {"bytes": 3 * 2 * (16 * kc + 8 * n), "flops": _transforms(n, 6)}
    if kind == "les":
        net = 10 * 64 + 64 * 64 + 64 * 6
        return {"bytes": 2 * 3 * 16 * kc, "flops": 4 * (_transforms(n, 8 + 9 + 6) + 2.0 * n * net)}
    fields = {"mhd": 6, "bouss": 3, "hydro": d}.get(case.get("physics"), 4)
    if kind == "generic3d":
        return {"bytes": 2 * fields * 16 * kc, "flops": 2 * _transforms(n, 3 + 12 + 4)}
    per_rhs = {("hydro", 3): 8, ("mhd", 3): 14, ("hydro", 2): 4, ("bouss", 2): 7}[(case["physics"], d)]
    stages = {"step3d": 4, "step2d": 2, "rhs3d": 1}[kind]
    return {"bytes": 2 * fields * 16 * kc, "flops": stages * _transforms(n, per_rhs)}


# ------------------------------------------------------------------ 64-bit values
def _project(f, ks):
    k2 = sum(k * k for k in ks)
    k2 = torch.where(k2 == 0, torch.ones_like(k2), k2)
    div = sum(k * c for k, c in zip(ks, f)) / k2
    return [c - k * div for k, c in zip(ks, f)]


def _rhs_exact(case, shape, closure=None):
    """f({field: k arrays}) -> {field: k arrays}: the right-hand side, 2/3 dealiased."""
    ks, keep, d = _kvec(shape), _kept(shape), len(shape)
    names = list(range(d))

    def fwd(x):
        return _fwd(x) * keep

    def grad(c):
        return [_bwd(1j * k * c, shape) for k in ks]

    def curl(a):
        return [1j * (ks[(i + 1) % 3] * a[(i + 2) % 3] - ks[(i + 2) % 3] * a[(i + 1) % 3]) for i in range(3)]

    def cross(a, b):
        return [a[(i + 1) % 3] * b[(i + 2) % 3] - a[(i + 2) % 3] * b[(i + 1) % 3] for i in range(3)]

    def rhs(s):
        u = s["u"]
        ux = [_bwd(c, shape) for c in u]
        du = []
        for c in u:
            g = grad(c)
            du.append(-fwd(sum(ux[i] * g[i] for i in names)))
            del g
        out = {}
        if case["kind"] == "generic3d":
            om = _OMEGA[::-1]
            du = [du[i] - 2 * (om[(i + 1) % 3] * u[(i + 2) % 3] - om[(i + 2) % 3] * u[(i + 1) % 3]) for i in range(3)]
        if "B" in s:
            bx = [_bwd(c, shape) for c in s["B"]]
            jx = [_bwd(c, shape) for c in curl(s["B"])]
            lor = cross(jx, bx)
            du = [a + fwd(b) / (4 * math.pi) for a, b in zip(du, lor)]
            out["B"] = curl([fwd(c) for c in cross(ux, bx)])
        if "T" in s:
            up = d - 1                                        # gravity along y in 2D, z in 3D
            du[up] = du[up] + s["T"][0]
            g = grad(s["T"][0])
            out["T"] = [-fwd(sum(ux[i] * g[i] for i in names)) - u[up]]
        if closure is not None:
            du = [a + b for a, b in zip(du, closure(u))]
        out["u"] = _project(du, ks)
        return out

    return rhs


def _phis(z):
    small = z.abs() < 0.5
    zs = torch.where(small, z, torch.zeros_like(z))
    zl = torch.where(small, -torch.ones_like(z), z)
    t1, t2 = torch.zeros_like(z), torch.zeros_like(z)
    for j in range(18, 0, -1):                                # sum z^(j-1)/j!, sum z^(j-2)/j!
        t1 = t1 * zs + 1.0 / math.factorial(j)
        if j > 1:
            t2 = t2 * zs + 1.0 / math.factorial(j)
    f1 = torch.where(small, t1, torch.expm1(zl) / zl)
    f2 = torch.where(small, t2, (torch.expm1(zl) / zl - 1) / zl)
    return torch.exp(z), f1, f2


def _advance_exact(y, rhs, coeff, shape, dt, scheme):
    """One exponential-time-differencing step; coeff: {field: diffusivity}."""
    k2 = sum(k * k for k in _kvec(shape))

    def etd1(a, n, h):
        out = {}
        for name in a:
            f0, f1, _ = _phis(-coeff[name] * k2 * h)
            out[name] = [c * f0 + b * (f1 * h) for c, b in zip(a[name], n[name])]
        return out

    def combine(terms):
        return {name: [sum(w * t[name][i] for w, t in terms) for i in range(len(y[name]))] for name in y}

    k1 = rhs(y)
    if scheme == "RK4":
        k2_ = rhs(etd1(y, k1, dt / 2))
        k3 = rhs(etd1(y, k2_, dt / 2))
        total = combine([(1 / 6.0, k1), (1 / 3.0, k2_), (1 / 3.0, k3)])
        k4 = rhs(etd1(y, k3, dt))
        return etd1(y, combine([(1.0, total), (1 / 6.0, k4)]), dt)
    if scheme == "RK2mid":
        kb = rhs(etd1(y, k1, dt / 2))
        out = etd1(y, k1, dt)
        weight = 2.0
    else:
        out = etd1(y, k1, dt)
        kb = rhs(out)
        weight = 1.0
    for name in y:
        _, _, f2 = _phis(-coeff[name] * k2 * dt)
        out[name] = [c + (b - a) * (weight * f2 * dt) for c, a, b in zip(out[name], k1[name], kb[name])]
    return out


def _closure_exact(shape):
    """The closure term of the LES with the shipped network, nothing rounded."""
    z = np.load(os.path.join(_ROOT, "dedalus-1.0_gb300", "data", "les_closure_256to64.npz"))
    p = torch.from_numpy(z["params"].astype(np.float64)).cuda()
    norm = torch.from_numpy(z["norm"].astype(np.float64)).cuda()
    norm[40:46] *= float(z["gain"])
    delta, table = float(z["delta"]), torch.from_numpy(z["shell_w"].astype(np.float64)).cuda()
    W1, b1, W2, b2, W3, b3 = (v.reshape(s) for v, s in zip(torch.split(p, [1024, 64, 4096, 64, 512, 8]), (
        (64, 16), (64,), (64, 64), (64,), (8, 64), (8,))))
    ks, keep = _kvec(shape), _kept(shape)
    kk = torch.sqrt(sum(k * k for k in ks))
    i = kk.floor().long().clamp(max=table.numel() - 2)
    w = torch.where(kk >= table.numel() - 1, table[-1], table[i] + (kk - i) * (table[i + 1] - table[i]))
    rows = [(0, 3, 4), (3, 1, 5), (4, 5, 2)]

    def term(u):
        g = [_bwd(1j * ks[j] * u[a], shape).reshape(-1) for a in range(3) for j in range(3)]
        x = torch.stack(g + [torch.full_like(g[0], delta)], 1)
        x = (x - norm[:10]) * norm[16:26]
        h = torch.tanh(torch.tanh(x @ W1[:, :10].T + b1) @ W2.T + b2)
        tau = (h @ W3[:6].T + b3[:6]) * norm[40:46] + norm[32:38]
        th = [_fwd(tau[:, c].reshape(shape)) * keep for c in range(6)]
        return [-w * sum(1j * ks[j] * th[rows[a][j]] for j in range(3)) for a in range(3)]

    return term


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        for slab, n in zip(_ensemble_inputs(case, seed), _CLASSES):
            rhs = _rhs_exact(dict(case, physics="bouss"), (n, n))
            runs = []
            for run_ in slab:
                y = _advance_exact({"u": [run_[0], run_[1]], "T": [run_[2]]}, rhs, {"u": 2e-3, "T": 2e-3}, (n, n), 1e-2,
                                   "RK2mid")
                runs.append(torch.stack(y["u"] + y["T"]))
            out.append(torch.stack(runs))
        return out
    if kind == "train":
        X, T, p = _train_inputs(case, seed)
        p = p.double().requires_grad_(True)
        W1, b1, W2, b2, W3, b3 = (v.reshape(s) for v, s in zip(torch.split(p, [1024, 64, 4096, 64, 512, 8]), (
            (64, 16), (64,), (64, 64), (64,), (8, 64), (8,))))
        h = torch.tanh(torch.tanh(X.double() @ W1.T + b1) @ W2.T + b2)
        e = ((h @ W3.T + b3)[:, :6] - T[:, :6].double())
        total = (e * e).sum()
        (total / (6.0 * case["samples"])).backward()
        return dict(grad=p.grad, loss=total.detach().reshape(1), params=None)
    if kind == "les":
        case = dict(case, nz=case["n"], ny=case["n"], nx=case["n"], physics="hydro")
    shape, y = _shape(case), _inputs(case, seed)
    if kind == "transform":
        return dict(x=[_bwd(c, shape) for c in y["u"]], k=y["u"])
    rhs = _rhs_exact(case, shape, _closure_exact(shape) if kind == "les" else None)
    if kind == "rhs3d":
        r = rhs(y)
        return {name: r[name] for name in y}
    coeff = {"bouss": {"u": 2e-3, "T": 2e-3}}.get(case.get("physics"), {"u": 5e-3, "B": 5e-3, "T": 5e-3})
    if kind == "step2d" and case["physics"] == "hydro":
        coeff = {"u": 1e-3}
    scheme = {"step2d": "RK2mid", "generic3d": "RK2trap"}.get(kind, "RK4")
    return _advance_exact(y, rhs, coeff, shape, _dt(case), scheme)
