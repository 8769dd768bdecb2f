"""The one-call 3D right-hand side in advective form (csrc/advect.cu) at the x lengths
that test_gpu_advect leaves out, with and without the scalar: 512 points with it
are the most that a block of thread groups holds (15 groups of two warps, all named
barriers).  Oracle and operator sequence, 1e-12 relative L2 per field as there.
"""
import numpy as np
import pytest

from oracle import physics as OP
from oracle import representation as OR

pytestmark = pytest.mark.gpu
OM = np.array([0.7, -0.2, 0.3])


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("name", ["IncompressibleHydro", "BoussinesqHydro"])
@pytest.mark.parametrize("shape", [(16, 16, 16), (16, 16, 24), (16, 16, 32), (16, 24, 48), (16, 16, 64), (24, 16, 96), (16, 16, 128),
                                   (16, 16, 192), (16, 16, 256), (16, 16, 512), (512, 16, 16), (16, 256, 16)])
def test_lengths(dd, cuda, name, shape):
    G = getattr(dd.mods, name)(shape, dd.mods.FourierRepresentation)
    S = getattr(dd.mods, name)(shape, dd.mods.FourierRepresentation)
    O = getattr(OP, name)(shape, OR.FourierRepresentation)
    for P in (G, S, O):
        P.parameters.update(Omega=OM)
        if name == "BoussinesqHydro":
            P.parameters.update(boussinesq_direction="z", beta=0.6, g=1.2)
    S._advect_fused = lambda data: False
    dg, do = G.create_fields(0.3), O.create_fields(0.3)
    rng = np.random.default_rng(12)
    for f, field in do:
        for i, c in field:
            k = np.transpose(np.fft.rfftn(rng.standard_normal(shape)), (1, 0, 2)) / np.prod(shape)
            c["kspace"] = k.copy()
            dg[f][i]["kspace"] = k
    ko, kg, ks = O.create_fields(0.), G.create_fields(0.), S.create_fields(0.)
    O.RHS(do, ko)
    G.RHS(dg, kg)
    assert G._advect_fused(dg)
    S.RHS(dg, ks)
    for f, field in ko:
        for i, c in field:
            a = kg[f][i].to_numpy("kspace")
            assert _rel(a, c["kspace"]) < 1e-12, (f, i)
            assert _rel(a, ks[f][i].to_numpy("kspace")) < 1e-12, (f, i)
