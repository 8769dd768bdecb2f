"""FP64 transforms of subnormal values (csrc/fft_fixed.cuh scales their pencils by a
power of two on the way in and back on the way out) against numpy in extended
precision.

Tolerance, in units u = 2^-1074 of the subnormal grid: every pass rounds each
component to it once (u/2).  A later pass over n values adds their errors with
factors of modulus one, so a component is off by at most n sqrt(2) u/2 from the pass before and
u/2 from its own rounding.  Forward: x pass, then n_y (and n_z) values; the backward
transform: (n_z, then) n_y values, then the n_x of the packed half spectra of two
rows.  numpy's error is far below u.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = np.ldexp(np.longdouble(1), -1074)
_SHAPES = [(16, 32), (48, 24), (8, 16, 64), (64, 8), (16, 512), (256, 32)]


def _field(dd, shape):
    M = dd.mods
    return M.IncompressibleHydro(shape, M.FourierRepresentation).create_fields(0.)["u"][0]


def _bound(ns):
    e = 0.5
    for n in ns:
        e = n * np.sqrt(2.0) * e + 0.5
    return e


@pytest.mark.parametrize("bits", [6, 20, 31])
@pytest.mark.parametrize("shape", _SHAPES)
def test_subnormal(dd, cuda, shape, bits):
    """Integers of up to `bits` bits in units of 2^-1074: high words all zero (the 20
    leading mantissa bits of a subnormal start at 2^32 units)."""
    rng = np.random.default_rng(bits)
    perm = (1, 0, 2) if len(shape) == 3 else (1, 0)
    unit = 5e-324
    x = rng.integers(-2 ** bits, 2 ** bits, shape).astype(np.float64) * unit
    assert np.abs(x).max() < 2.0 ** -1042 and np.any(x)
    c = _field(dd, shape)
    c["xspace"] = x
    k = c.to_numpy("kspace").copy()
    ref = np.transpose(np.fft.rfftn(x.astype(np.longdouble) / U) / np.longdouble(x.size), perm)
    kx, kt = np.arange(shape[-1] // 2 + 1), [np.abs(np.fft.fftfreq(n) * n) for n in shape[:-1]]
    keep = kx < shape[-1] / 3                              # 2/3 rule, k-layout
    if len(shape) == 3:
        keep = (kt[1] < shape[1] / 3)[:, None, None] & (kt[0] < shape[0] / 3)[None, :, None] & keep[None, None, :]
    else:
        keep = keep[:, None] & (kt[0] < shape[0] / 3)[None, :]
    got = k.view(np.float64).astype(np.longdouble).view(np.clongdouble) / U
    e = np.abs(got - np.where(keep, ref, 0))
    assert e.max() <= np.sqrt(2.0) * _bound(shape[-2::-1])
    # backward, from a spectrum of integers
    k = np.where(keep, rng.integers(-2 ** bits, 2 ** bits, k.shape) + 1j * rng.integers(-2 ** bits, 2 ** bits, k.shape), 0)
    if bits == 6:
        k.real[keep] = 1                                   # one unit everywhere
    c["kspace"] = (k.view(np.float64) * unit).view(np.complex128)
    back = c.to_numpy("xspace").astype(np.longdouble) / U
    a = np.transpose(k.astype(np.clongdouble), perm)
    for ax in range(len(shape) - 1):
        a = np.fft.ifft(a, axis=ax) * shape[ax]
    ref = np.fft.irfft(a, n=shape[-1], axis=-1) * shape[-1]
    assert np.any(np.abs(ref) > 1)
    # a value of the row pass: kx >= 0 entries count twice, for two rows packed in one pencil
    bound = 2 * shape[-1] * np.sqrt(2.0) * (_bound(shape[:-2]) * shape[-2] * np.sqrt(2.0) + 0.5) + 0.5
    assert np.abs(back - ref).max() <= bound
