"""The q tables (1/k^2 and phi functions per integer k^2) cover every mode of the
grids that use them: boxes of sides 2 pi / m have integer wavenumbers up to m N/2,
not N/2.  Table sizes on the CPU; steps on such boxes against the oracle on the
GPU, 1e-12 relative L2 per step as for the other boxes."""
import types

import numpy as np
import pytest

from oracle import physics as OP, time_step as OT
from oracle.representation import FourierRepresentation as OracleRep

P = np.pi
_BOXES = [((64, 64, 64), (P, P, P)), ((16, 32, 8), (2 * P, P, P / 2)), ((32, 64), (P, 2 * P)), ((128, 128), (P / 4, P / 4)),
          ((64, 64, 64), (2 * P, 2 * P, 2 * P)), ((512, 512, 512), (2 * P, 2 * P, 2 * P))]


def _k2_max(dd, shape, length):
    k, _, _ = dd.kgrid.wavenumbers(shape, length)
    return sum(np.max(np.abs(v)) ** 2 for v in k.values())


@pytest.mark.parametrize("shape,length", _BOXES)
def test_tables_cover_the_grid(dd, monkeypatch, shape, length):
    q = _k2_max(dd, shape, length)
    assert dd.kgrid.integer_k(shape, length)
    plan = types.SimpleNamespace(xshape=shape, ndim=len(shape), device="cpu",
                                 integer_k2_max=dd.kgrid.integer_k2_max(shape, length), integer_k=True)
    phys = dd.mods.IncompressibleHydro(shape, dd.mods.FourierRepresentation, length=length)
    sizes = []
    monkeypatch.setattr(dd.physics._lib, "call", lambda name, nd, nu, vo, h, qmax, t, st: sizes.append(qmax))
    monkeypatch.setattr(dd.physics, "current_stream", lambda: None)
    assert phys.inv_k2_table(plan).numel() == q + 1
    t = phys.phi_table(plan, 1e-3, 1, 1e-3)
    assert sizes == [q] and t.shape == (q + 1, 4)


@pytest.mark.parametrize("shape,length,use", [((32, 32), (1.5, 2 * P), False), ((32, 32), (4 * P, 2 * P), False),
                                              ((64, 64), (2 * P / 45, 2 * P / 45), True),    # 2 (45 32)^2 = 4147200
                                              ((64, 64), (2 * P / 46, 2 * P / 46), False)])  # 2 (46 32)^2 = 4333568
def test_boxes_without_tables(dd, shape, length, use):
    assert dd.kgrid.integer_k(shape, length) == use
    if use:
        assert dd.kgrid.integer_k2_max(shape, length) == _k2_max(dd, shape, length) <= dd.kgrid.INTEGER_K2_LIMIT


def _pair(dd, cls, shape, length, params, fields):
    M = dd.mods
    out = []
    for r in (getattr(OP, cls)(shape, OracleRep, length=length), getattr(M, cls)(shape, M.FourierRepresentation, length=length)):
        r.parameters.update(params)
        d = r.create_fields(0.)
        for (f, c), a in fields.items():
            d[f][c]["kspace"] = a.copy()
        out.append((r, d))
    return out


def _rel(dg, do):
    a = [(c.to_numpy("kspace"), do[f][i]["kspace"]) for f, field in dg for i, c in field]
    return np.sqrt(sum(np.sum(np.abs(g - r) ** 2) for g, r in a) / sum(np.sum(np.abs(r) ** 2) for g, r in a))


@pytest.mark.gpu
@pytest.mark.parametrize("shape,length", [((32, 32, 32), (P, P, P)), ((16, 32, 48), (2 * P, P, P / 2)), ((64, 32), (P, P)),
                                          ((64, 64), (2 * P / 46, 2 * P / 46))])
def test_steps_match_oracle(dd, cuda, shape, length):
    M, nd = dd.mods, len(shape)
    init = dd.init_cond.turbulence_3d if nd == 3 else dd.init_cond.turbulence_2d
    u = init(shape, length=length, seed=41, k0=4.0 * 2 * P / min(length))
    (ro, do), (rg, dg) = _pair(dd, "IncompressibleHydro", shape, length, {"nu": 1e-4}, {("u", i): u[i] for i in range(nd)})
    to, tg = (OT.RK4(ro), M.RK4(rg)) if nd == 3 else (OT.RK2mid(ro), M.RK2mid(rg))
    for _ in range(2):
        to.do_advance(do, 1e-3)
        tg.do_advance(dg, 1e-3)
    assert _rel(dg, do) < 1e-12


@pytest.mark.gpu
def test_energy_outside_the_kept_modes(dd, cuda):
    """The decay of modes outside the kept set reads the tables up to the corner of the grid."""
    shape, length = (32, 16, 32), (P, P, P)
    rng = np.random.default_rng(5)
    f = {("u", i): np.transpose(np.fft.rfftn(rng.standard_normal(shape)), (1, 0, 2)) / np.prod(shape) for i in range(3)}
    (ro, do), (rg, dg) = _pair(dd, "IncompressibleHydro", shape, length, {"nu": 1e-3}, f)
    OT.RK4(ro).do_advance(do, 1e-3)
    dd.mods.RK4(rg).do_advance(dg, 1e-3)
    assert _rel(dg, do) < 1e-12
