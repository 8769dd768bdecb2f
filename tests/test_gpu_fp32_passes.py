"""FP32 y and z passes at the lengths with narrow tiles (16 pencils), on rows that
keep fewer modes than a tile, exactly one tile, two tiles and a ragged number,
against the CPU oracle.  Tolerance: three passes of at most three radices, each a
rounding of 2^-24 on up to 4 levels of additions and one twiddle product, amount
to at most 3 * 3 * 5 * 2^-24 = 2.7e-6 in the worst direction; errors of random
sign stay below 2e-6, the tolerance of the other FP32 transforms.
"""
import numpy as np
import pytest

from oracle import representation as OR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [16, 48, 96, 128])
@pytest.mark.parametrize("nz,ny", [(32, 48), (48, 32), (96, 128), (128, 96)])
def test_matches_oracle(dd, cuda, nz, ny, nx):
    import torch
    shape = (nz, ny, nx)
    rep = OR.FourierRepresentation(None, shape, (2 * np.pi,) * 3)
    x = np.random.default_rng(nx).standard_normal(shape)
    rep['xspace'] = x
    k = rep['kspace'].copy()
    plan = dd.engine.Plan(shape, (2 * np.pi,) * 3)
    kd = torch.zeros(plan.kshape, dtype=torch.complex128, device=cuda)
    plan.r2c([torch.from_numpy(x).to(cuda)], [kd], precision=dd._lib.DD_FP32)
    assert np.linalg.norm(kd.cpu().numpy() - k) < 2e-6 * np.linalg.norm(k)
    rep['kspace'] = k
    back = rep['xspace'].copy()
    xd = torch.empty(shape, dtype=torch.float64, device=cuda)
    plan.c2r([torch.from_numpy(k).to(cuda)], [xd], precision=dd._lib.DD_FP32)
    assert np.linalg.norm(xd.cpu().numpy() - back) < 2e-6 * np.linalg.norm(back)
