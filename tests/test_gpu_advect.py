"""The one-call 3D right-hand side in advective form (csrc/advect.cu: rotation,
Boussinesq, static basis) against the CPU oracle and against the operator
sequence it stands for, with energy outside the kept modes in the state (only the
linear terms act there).  Tolerance: as for the operator sequence, 1e-12 relative
L2 per field (the FFT algorithms differ, every other operation is rounded alike).
"""
import numpy as np
import pytest

from oracle import physics as OP
from oracle import representation as OR

pytestmark = pytest.mark.gpu

_CASES = [
    ("IncompressibleHydro", (16, 24, 32), {"nu": 1e-2, "Omega": np.array([0.7, -0.2, 0.3])}),
    ("IncompressibleHydro", (96, 16, 48), {"Omega": np.array([0.0, 0.0, 1.0])}),
    ("BoussinesqHydro", (48, 32, 16), {"nu": 2e-3, "kappa": 1e-3, "g": 1.3, "alpha_t": 0.7, "beta": 0.4,
                                       "boussinesq_direction": "x"}),
    ("BoussinesqHydro", (16, 64, 24), {"nu": 2e-3, "kappa": 2e-3, "Omega": np.array([0.1, 0.2, -0.5]),
                                       "boussinesq_direction": "y"}),
    ("BoussinesqHydro", (16, 16, 192), {"beta": -1.5, "boussinesq_direction": "z"}),
    ("BoussinesqHydro", (8, 16, 16), {"nu": 2e-3, "boussinesq_direction": "z"}),     # below the fused lengths
]


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("name,shape,params", _CASES)
def test_matches_oracle_and_operator_sequence(dd, cuda, monkeypatch, name, shape, params):
    G = getattr(dd.mods, name)(shape, dd.mods.FourierRepresentation)
    O = getattr(OP, name)(shape, OR.FourierRepresentation)
    for P in (G, O):
        P.parameters.update(params)
    dg, do = G.create_fields(0.3), O.create_fields(0.3)
    rng = np.random.default_rng(11)
    for f, field in do:
        for i, c in field:
            k = np.transpose(np.fft.rfftn(rng.standard_normal(shape)), (1, 0, 2)) / np.prod(shape)
            c["kspace"] = k.copy()
            dg[f][i]["kspace"] = k
    ko, kg, ks = O.create_fields(0.), G.create_fields(0.), G.create_fields(0.)
    O.RHS(do, ko)
    G.RHS(dg, kg)
    assert G._advect_fused(dg) == (min(shape) >= 16)
    monkeypatch.setattr(type(G), "_advect_fused", lambda self, data: False)
    G.RHS(dg, ks)
    assert kg.time == 0.3
    for f, field in ko:
        for i, c in field:
            a = kg[f][i].to_numpy("kspace")
            assert _rel(a, c["kspace"]) < 1e-12, (f, i)
            assert _rel(a, ks[f][i].to_numpy("kspace")) < 1e-12, (f, i)
