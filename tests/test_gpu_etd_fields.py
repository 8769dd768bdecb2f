"""dd_etd_fields gives, bit for bit, what dd_etd1 / dd_etd2rk1 / dd_etd2rk2 give
field by field: factors shared by consecutive fields, different ones, zeros and
NaN, more fields than one launch takes, and sizes around a block."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("n,nf", [(1, 1), (127, 3), (129, 4), (4099, 6), (3000, 7), (1 << 21, 2)])
def test_matches_single_fields(dd, cuda, ndim, n, nf):
    import torch
    L, dt = dd._lib, 0.05
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    g = torch.Generator(device=cuda).manual_seed(n + nf)
    s, d1, d2 = (torch.randn(nf, n, dtype=torch.complex128, device=cuda, generator=g) for _ in range(3))
    rng = np.random.default_rng(n)
    f = -np.abs(rng.standard_normal((nf, n))) * rng.choice([0., 0.1, 1., 30., 1e3], (nf, n))
    f[1:nf // 2 + 1] = f[0]                                # shared by the first fields
    if n > 1:
        f[-1, 1] = np.nan
        f[0, 2:9] = 0.
    f = torch.from_numpy(f).to(cuda)

    def p(t):
        return ctypes.c_void_p(t.data_ptr())

    def rows(t):
        return (ctypes.c_void_p * nf)(*[t[i].data_ptr() for i in range(nf)])

    for scheme, name in enumerate(("dd_etd1", "dd_etd2rk1", "dd_etd2rk2")):
        ref = torch.empty_like(s)
        for i in range(nf):
            d = (p(d1[i]),) if scheme == 0 else (p(d1[i]), p(d2[i]))
            L.call(name, ndim, p(s[i]), p(ref[i]), *d, p(f[i]), dt, n, st)
        out = s.clone()                                    # in place, as the integrators call it
        L.call("dd_etd_fields", ndim, scheme, nf, rows(out), rows(out), rows(d1), rows(d2) if scheme else None,
               rows(f), dt, n, st)
        assert torch.equal(torch.view_as_real(out).view(torch.int64), torch.view_as_real(ref).view(torch.int64))


def test_bad_arguments(dd, cuda):
    import torch
    t = torch.zeros(4, dtype=torch.complex128, device=cuda)
    f = torch.zeros(4, dtype=torch.float64, device=cuda)
    one, fac, none = ((ctypes.c_void_p * 1)(x) for x in (t.data_ptr(), f.data_ptr(), None))
    for args in ((4, 0, 1, one, one, one, None, fac), (3, 3, 1, one, one, one, one, fac),
                 (3, 1, 1, one, one, one, None, fac), (3, 1, 1, one, one, one, none, fac)):
        with pytest.raises(ValueError):
            dd._lib.call("dd_etd_fields", *args, 0.1, 4, None)
