"""Plans that keep the mode kx = Nx/2 (mx = Nx/2, no 2/3 rule along x): the C ABI
accepts them, the Python bounds never make one.  Transforms (FP64 and FP32) and
fused FP64 right-hand sides on such plans against numpy.

Tolerances (relative L2): single FP64 transforms as in test_gpu_fixed_transforms
(3.8e-16 for three passes); FP32 ones 1e-6 (0.6 u log2 N of the butterflies, u =
2^-24: 6.8e-7 at the largest N here, 2^19); right-hand sides, whose
derivatives and projection act on transform errors of that size, 1e-12, as the
other right-hand side tests.
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = {0: 3.8e-16, 1: 1e-6}
RHS_TOL = 1e-12
_LENS = [8, 16, 24, 32, 48, 64, 96, 128, 192, 256, 512]


def _rel(a, b):
    return float(np.sqrt(np.sum(np.abs(a - b) ** 2) / np.sum(np.abs(b) ** 2)))


class _Plan:
    """A native plan that keeps every mode but the Nyquist ones of y and z."""

    def __init__(self, dd, shape):
        self.dd, self.shape, self.nd = dd, shape, len(shape)
        kg = dd.kgrid
        self.k = kg.k_tables(shape, (2 * np.pi,) * self.nd)
        self.kshape = kg.kspace_shape(list(shape))
        nx, ny, nz = shape[-1], shape[-2], (shape[0] if self.nd == 3 else 2)
        p = [None if t is None else t.ctypes.data_as(ctypes.c_void_p) for t in self.k]
        self.h = ctypes.c_void_p()
        dd._lib.call("dd_plan_create", self.nd, (ctypes.c_int64 * self.nd)(*shape), *p, nx // 2, ny // 2 - 1, nz // 2 - 1,
                     ctypes.byref(self.h))
        # kept mask in k-layout
        full = [np.abs(np.fft.fftfreq(n) * n) < n / 2 for n in (ny, nz)]
        x = np.ones(nx // 2 + 1, dtype=bool)
        self.mask = (full[0][:, None, None] & full[1][None, :, None] & x[None, None, :] if self.nd == 3
                     else x[:, None] & full[0][None, :])

    def close(self):
        self.dd._lib.call("dd_plan_destroy", self.h)

    # numpy transforms between the k-layout and grid points, in the operands' precision
    def forward(self, x):
        k = np.fft.rfftn(x, axes=tuple(range(self.nd))) / np.longdouble(x.size)
        return np.where(self.mask, np.transpose(k, (1, 0, 2) if self.nd == 3 else (1, 0)), 0)

    def backward(self, k):
        k = np.transpose(np.where(self.mask, k, 0), (1, 0, 2) if self.nd == 3 else (1, 0))
        for a in range(self.nd - 1):
            k = np.fft.ifft(k, axis=a) * self.shape[a]
        return np.fft.irfft(k, n=self.shape[-1], axis=-1) * self.shape[-1]

    def axes(self):
        kx, ky, kz = self.k
        return ([kx[None, None, :], ky[:, None, None], kz[None, :, None]] if self.nd == 3
                else [kx[:, None], ky[None, :]])

    # the library's transforms
    def _ws(self, prec):
        n = ctypes.c_size_t()
        self.dd._lib.call("dd_plan_workspace_size", self.h, 1, prec, ctypes.byref(n))
        return torch.empty(n.value, dtype=torch.uint8, device="cuda")

    def fft(self, name, a, out, prec):
        ws = self._ws(prec)
        ap, _a = self.dd._lib.ptr_array([a.data_ptr()])
        op, _o = self.dd._lib.ptr_array([out.data_ptr()])
        self.dd._lib.call(name, self.h, 1, ap, op, prec, ctypes.c_void_p(ws.data_ptr()), ws.numel(),
                          self.dd.engine.current_stream())
        return out.cpu().numpy()


def _spectrum(p, rng, real):
    """Random spectrum on all modes; real: of a real field (Hermitian)."""
    if real:
        return p.forward(rng.standard_normal(p.shape)).astype(np.complex128)
    return rng.standard_normal(p.kshape) + 1j * rng.standard_normal(p.kshape)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", _LENS)
def test_transforms(dd, cuda, n, prec):
    for shape in [(8, 16, n), (24, n)]:
        p = _Plan(dd, shape)
        rng = np.random.default_rng(n)
        k = _spectrum(p, rng, False)
        ref = p.backward(k.astype(np.clongdouble))
        assert np.abs(np.fft.rfft(ref.astype(np.float64), axis=-1)[..., -1]).max() > 0    # the mode is there
        x = p.fft("dd_fft_c2r", torch.from_numpy(k).cuda(), torch.empty(shape, dtype=torch.float64, device="cuda"), prec)
        assert _rel(x, ref) < TOL[prec]
        kk = p.fft("dd_fft_r2c", torch.from_numpy(x).cuda(), torch.empty(p.kshape, dtype=torch.complex128, device="cuda"),
                   prec)
        assert _rel(kk, p.forward(x.astype(np.longdouble))) < TOL[prec]
        p.close()


@pytest.mark.parametrize("p2", [-900, 60])
def test_prescaled_values(dd, cuda, p2):
    """The mode alone, and beside others, where pencils are pre-scaled (below 2^-895, above 2^49)."""
    p = _Plan(dd, (16, 32))
    rng = np.random.default_rng(4)
    k = np.zeros(p.kshape, dtype=np.complex128)
    k[16] = rng.standard_normal(16) + 1j * rng.standard_normal(16)
    for a in (k, _spectrum(p, rng, False)):
        x = [p.fft("dd_fft_c2r", torch.from_numpy(np.ldexp(a.view(np.float64), e).view(np.complex128)).cuda(),
                   torch.empty(p.shape, dtype=torch.float64, device="cuda"), 0) for e in (0, p2)]
        assert np.any(x[0]) and np.array_equal(np.ldexp(x[0], p2), x[1])
    p.close()


def test_shear_backward(dd, cuda):
    """dd_shear_c2r without shear and with no cut along y is dd_fft_c2r."""
    for shape in [(16, 32), (8, 16, 24)]:
        p = _Plan(dd, shape)
        nh, ny = shape[-1] // 2 + 1, shape[-2]
        k = torch.from_numpy(np.where(p.mask, _spectrum(p, np.random.default_rng(2), False), 0)).cuda()
        # ky per (ky, kx) in k order, the Nyquist row beyond the cut as the plan has it
        ky = np.abs(p.k[1])
        kys = np.broadcast_to(ky[:, None] if len(shape) == 3 else ky[None, :],
                              (ny, nh) if len(shape) == 3 else (nh, ny))
        kys = torch.from_numpy(np.ascontiguousarray(kys)).cuda()
        pr = torch.zeros((ny, nh), dtype=torch.float64, device="cuda")
        x = torch.empty(shape, dtype=torch.float64, device="cuda")
        n = ctypes.c_size_t()
        dd._lib.call("dd_shear_workspace_size", p.h, 1, ctypes.byref(n))
        ws = torch.empty(n.value, dtype=torch.uint8, device="cuda")
        kp, _a = dd._lib.ptr_array([k.data_ptr()])
        xp, _b = dd._lib.ptr_array([x.data_ptr()])
        dd._lib.call("dd_shear_c2r", p.h, 1, kp, xp, ctypes.c_void_p(kys.data_ptr()), float(ny // 2),
                     ctypes.c_void_p(pr.data_ptr()), 0.0, ctypes.c_void_p(ws.data_ptr()), ws.numel(),
                     dd.engine.current_stream())
        assert _rel(x.cpu().numpy(), p.backward(k.cpu().numpy().astype(np.clongdouble))) < TOL[0]
        p.close()


def _project(p, N):
    k = p.axes()
    k2 = sum(a ** 2 for a in k)
    ph = sum(a * n for a, n in zip(k, N)) / np.where(k2 == 0, 1, k2)
    return [n - a * ph for a, n in zip(k, N)]


def _rhs_rotational(p, u):
    """P[u x curl u]."""
    k, x = p.axes(), [p.backward(c) for c in u]
    d = lambda c, a: 1j * k[a] * u[c]
    if p.nd == 2:
        w = p.backward(d(1, 0) - d(0, 1))
        N = [x[1] * w, -x[0] * w]
    else:
        w = [p.backward(d((a + 2) % 3, (a + 1) % 3) - d((a + 1) % 3, (a + 2) % 3)) for a in range(3)]
        N = [x[(a + 1) % 3] * w[(a + 2) % 3] - x[(a + 2) % 3] * w[(a + 1) % 3] for a in range(3)]
    return _project(p, [p.forward(n) for n in N])


def _rhs_advective(p, u):
    """P[-(u . grad) u]."""
    k, x = p.axes(), [p.backward(c) for c in u]
    N = [-sum(p.backward(1j * k[a] * c) * x[a] for a in range(p.nd)) for c in u]
    return _project(p, [p.forward(n) for n in N])


def _call_rhs(p, u, kind):
    lib = p.dd._lib
    t = [torch.from_numpy(c).cuda() for c in u]
    o = [torch.full(p.kshape, float("nan"), dtype=torch.complex128, device="cuda") for _ in u]
    tp, _a = lib.ptr_array([c.data_ptr() for c in t])
    op, _b = lib.ptr_array([c.data_ptr() for c in o])
    n, st = ctypes.c_size_t(), p.dd.engine.current_stream()
    if kind == "advect":
        lib.call("dd_advect_workspace_size", p.h, 0, ctypes.byref(n))
    else:
        lib.call("dd_rhs%dd_workspace_size" % p.nd, p.h, *((1,) if p.nd == 2 else (0,)), 0, ctypes.byref(n))
    ws = torch.empty(n.value, dtype=torch.uint8, device="cuda")
    w = (ctypes.c_void_p(ws.data_ptr()), ws.numel(), st)
    if kind == "advect":
        lib.call("dd_advect_rhs3d", p.h, 0, None, None, tp, op, *w)
    elif p.nd == 2:
        lib.call("dd_rhs2d", p.h, 0, None, 1, tp, 0, op, 0, None, 0, 1, *w)
    else:
        lib.call("dd_rhs3d", p.h, 0, None, tp, op, None, 0, 1, *w)
    return [c.cpu().numpy() for c in o]


_SHAPES2 = [(32, 32), (48, 64), (32, 96), (64, 192), (32, 256), (32, 512)]
_SHAPES3 = [(16, 16, 16), (16, 24, 48), (16, 16, 64), (16, 16, 128)]


@pytest.mark.parametrize("shape,kind", [(s, "rotational") for s in _SHAPES2 + _SHAPES3] + [(s, "advect") for s in _SHAPES3])
def test_fused_right_hand_sides(dd, cuda, shape, kind):
    p = _Plan(dd, shape)
    rng = np.random.default_rng(7)
    u = [_spectrum(p, rng, True) for _ in shape]
    ref = (_rhs_advective if kind == "advect" else _rhs_rotational)(p, u)
    got = _call_rhs(p, u, kind)
    for a, b in zip(got, ref):
        assert _rel(a, np.where(p.mask, b, 0)) < RHS_TOL
    p.close()
