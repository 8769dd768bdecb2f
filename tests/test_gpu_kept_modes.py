"""FP64 and FP32 forward transforms write every mode that the dealiasing rule keeps
and exact zeros elsewhere, at every length along every axis.  The mask comes from the
rule itself (|m| < N/3 for 2/3; |m| < N/2 for 'None'), not from the result.
Tolerances, relative L2: FP64 as in test_gpu_fixed_transforms; FP32 0.6 u log2 N
of the butterflies with u = 2^-24, below 1e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {"fp64": 3.8e-16, "fp32": 1e-6}
_LENS = [8, 16, 24, 32, 48, 64, 96, 128, 192, 256, 512]
_SHAPES = sorted({s for n in _LENS for s in ((16, 8, n), (8, n, 24), (n, 24, 8), (n, 16), (32, n))})


def _mask(shape, rule):
    """Kept modes in k-layout (ky, kz, kx) or (kx, ky)."""
    part = 3 if rule == "2/3 cython" else 2
    ax = [np.abs(np.fft.fftfreq(n) * n).round() * part < n for n in shape[:-1]] + [np.arange(shape[-1] // 2 + 1) * part < shape[-1]]
    if len(shape) == 3:
        return ax[1][:, None, None] & ax[0][None, :, None] & ax[2][None, None, :]
    return ax[1][:, None] & ax[0][None, :]


@pytest.fixture(params=["2/3 cython", "None"])
def rule(dd, request):
    before = dd.config.decfg.get("FFT", "dealiasing")
    dd.config.decfg.set("FFT", "dealiasing", request.param)
    yield request.param
    dd.config.decfg.set("FFT", "dealiasing", before)


@pytest.mark.parametrize("shape", _SHAPES)
def test_forward(dd, cuda, rule, shape):
    import torch
    M = dd.mods
    c = M.IncompressibleHydro(shape, M.FourierRepresentation).create_fields(0.)["u"][0]
    assert c.plan.dealiasing == rule
    x = np.random.default_rng(sum(shape)).standard_normal(shape)
    ref = np.transpose(np.fft.rfftn(x.astype(np.longdouble)) / x.size, (1, 0, 2) if len(shape) == 3 else (1, 0))
    mask = _mask(shape, rule)
    ref = np.where(mask, ref, 0)
    for name, prec in (("fp64", 0), ("fp32", 1)):
        k = torch.full(c.kdata.shape, float("nan"), dtype=torch.complex128, device="cuda")
        c.plan.r2c([torch.from_numpy(x).cuda()], [k], precision=prec)
        k = k.cpu().numpy()
        assert not np.any(k[~mask])
        assert np.all(k[mask] != 0)
        assert np.sqrt(np.sum(np.abs(k - ref) ** 2) / np.sum(np.abs(ref) ** 2)) < TOL[name]


@pytest.mark.parametrize("shape", _SHAPES)
def test_backward(dd, cuda, rule, shape):
    """Every kept mode reaches the grid points, and nothing else does."""
    import torch
    M = dd.mods
    c = M.IncompressibleHydro(shape, M.FourierRepresentation).create_fields(0.)["u"][0]
    rng = np.random.default_rng(sum(shape))
    k = rng.standard_normal(tuple(c.kdata.shape)) + 1j * rng.standard_normal(tuple(c.kdata.shape))
    a = np.transpose(np.where(_mask(shape, rule), k, 0).astype(np.clongdouble), (1, 0, 2) if len(shape) == 3 else (1, 0))
    for ax in range(len(shape) - 1):
        a = np.fft.ifft(a, axis=ax) * shape[ax]
    ref = np.fft.irfft(a, n=shape[-1], axis=-1) * shape[-1]
    for name, prec in (("fp64", 0), ("fp32", 1)):
        x = torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")
        c.plan.c2r([torch.from_numpy(k).cuda()], [x], precision=prec)
        assert np.sqrt(np.sum((x.cpu().numpy() - ref) ** 2) / np.sum(ref ** 2)) < TOL[name]
