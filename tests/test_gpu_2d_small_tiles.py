"""Single 2D runs with 256- and 512-point y passes (tiles of 2 pencils) on rows
that keep an odd and an even number of modes, against the CPU oracle.  Tolerances:
those of the other right-hand sides, 1e-12 relative L2 in FP64 and 1e-4 with
FP32 transforms.
"""
import numpy as np
import pytest

from oracle import physics as OP
from oracle.representation import FourierRepresentation as OracleRep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-4)])
@pytest.mark.parametrize("shape", [(256, 32), (256, 64), (512, 32), (512, 128)])
def test_boussinesq_rhs(dd, cuda, shape, precision, tol):
    params = {'nu': 2e-3, 'kappa': 2e-3, 'g': 1., 'alpha_t': 1., 'beta': 1., 'boussinesq_direction': 'y'}
    u = dd.init_cond.turbulence_2d(shape, seed=4)
    fields = {('u', 0): u[0], ('u', 1): u[1], ('T', 0): dd.init_cond.band_limited_noise_2d(shape, seed=3)}
    dd.config.decfg.set('FFT', 'precision', precision)
    try:
        ro = OP.BoussinesqHydro(shape, OracleRep)
        rg = dd.mods.BoussinesqHydro(shape, dd.mods.FourierRepresentation)
        out = []
        for r in (ro, rg):
            r.parameters.update(params)
            d, e = r.create_fields(0.), r.create_fields(0.)
            for (name, i), a in fields.items():
                d[name][i]['kspace'] = a.copy()
            r.RHS(d, e)
            out.append(e)
    finally:
        dd.config.decfg.set('FFT', 'precision', 'fp64')
    for name, i in fields:
        ref = out[0][name][i]['kspace']
        assert np.linalg.norm(out[1][name][i].to_numpy('kspace') - ref) < tol * np.linalg.norm(ref)
