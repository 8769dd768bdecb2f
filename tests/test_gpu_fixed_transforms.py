"""FP64 transforms in block fixed point (csrc/fft_fixed.cuh) against numpy in
extended precision, at every supported length and at the edges of their
scaling: noise, one dominant mode, values scaled by powers of two into the
pre-scaled range, zeros, infinities and NaN.

Tolerance: each pass rounds its result to FP64 once (relative 2^-53 at most,
rms below 2^-53 / sqrt 3 of the values) and adds fixed-point errors of a few
units of 2^-62 of the pencil's bound, at most as much again; three passes stay
below 3 x 2^-53 x 2 / sqrt 3 = 3.8e-16 relative L2.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 3.8e-16
_LENS = [8, 16, 24, 32, 48, 64, 96, 128, 192, 256, 512]


def _field(dd, shape):
    M = dd.mods
    return M.IncompressibleHydro(shape, M.FourierRepresentation).create_fields(0.)["u"][0]


def _perm(shape):
    return (1, 0, 2) if len(shape) == 3 else (1, 0)


def _forward(c, x):
    c["xspace"] = x
    return c.to_numpy("kspace").copy()


def _backward(c, k):
    c["kspace"] = k
    return c.to_numpy("xspace").copy()


def _rel(a, b):
    return float(np.sqrt(np.sum(np.abs(a - b) ** 2) / np.sum(np.abs(b) ** 2)))


def _data(rng, shape, kind):
    x = rng.standard_normal(shape)
    if kind == "dominant":      # noise 12 decades below one mode
        g = np.meshgrid(*[np.arange(n) * 2 * np.pi / n for n in shape], indexing="ij")
        x = np.cos(sum(g)) + 1e-12 * x
    return x


@pytest.mark.parametrize("kind", ["noise", "dominant"])
@pytest.mark.parametrize("n", _LENS)
def test_lengths(dd, cuda, n, kind):
    shape = (8, 24, n) if n <= 64 else (n, 16)
    rng = np.random.default_rng(n)
    for s in {shape, shape[::-1]}:
        c = _field(dd, s)
        x = _data(rng, s, kind)
        k = _forward(c, x)
        ref = np.transpose(np.fft.rfftn(x.astype(np.longdouble)) / np.longdouble(x.size), _perm(s))
        keep = k != 0
        assert keep.sum() > 0.2 * k.size
        assert _rel(k, np.where(keep, ref, 0)) < TOL
        back = np.fft.irfftn(np.transpose(k.astype(np.clongdouble) * np.longdouble(x.size), _perm(s)), s=s,
                             axes=tuple(range(len(s))))
        assert _rel(_backward(c, k), back) < TOL


@pytest.mark.parametrize("p", [-960, -895, -700, 49, 51, 300, 900, 1000])
def test_powers_of_two_scale_exactly(dd, cuda, p):
    """x 2^p gives the transform times 2^p, bit for bit, also where the values
    are pre-scaled (below 2^-895, above 2^49)."""
    shape = (32, 48)
    rng = np.random.default_rng(5)
    c = _field(dd, shape)
    x = rng.standard_normal(shape)
    k = _forward(c, x)
    assert np.array_equal(_forward(c, np.ldexp(x, p)).view(np.float64), np.ldexp(k.view(np.float64), p))
    b = _backward(c, k)
    assert np.array_equal(_backward(c, np.ldexp(k.view(np.float64), p).view(np.complex128)), np.ldexp(b, p))


def test_rows_of_unequal_size(dd, cuda):
    """Two real rows share a pencil: a row 30 decades smaller stays within the
    rounding of the larger one, and zero rows beside zero rows stay zero."""
    shape = (16, 64)
    rng = np.random.default_rng(6)
    c = _field(dd, shape)
    x = rng.standard_normal(shape) * np.where(np.arange(16) % 2, 1e-30, 1.0)[:, None]
    ref = np.transpose(np.fft.rfftn(x.astype(np.longdouble)) / x.size, (1, 0))
    k = _forward(c, x)
    assert _rel(k, np.where(k != 0, ref, 0)) < TOL
    assert not np.any(_forward(c, np.zeros(shape)))
    assert not np.any(_backward(c, np.zeros_like(k)))


def test_overflow_and_not_finite(dd, cuda):
    shape = (16, 32)
    c = _field(dd, shape)
    k = np.zeros((17, 16), dtype=np.complex128)
    k[0, 0], k[1, 0] = 1.7e308, 0.5e308          # the sum at x = 0 leaves FP64's range
    b = _backward(c, k)
    ref = 1.7e308 * (1 + 2 * (0.5 / 1.7) * np.cos(np.arange(32) * 2 * np.pi / 32).astype(np.longdouble))
    fits = ref < np.finfo(np.float64).max
    assert np.all(np.isinf(b[:, ~fits])) and fits.sum() > 4
    assert np.max(np.abs(b[:, fits] / ref[fits] - 1)) < 1e-15
    for bad in (np.nan, np.inf):
        x = np.ones(shape)
        x[3, 5] = bad
        k = _forward(c, x)
        assert not np.any(np.isfinite(k[:11, :6])) and not np.any(k[11:])
