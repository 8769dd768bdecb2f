"""Work fields (aux_fields) after the one-call 3D rotating and Boussinesq right-hand
sides: there, with the time and the values that the operator sequence leaves, and
fields that it zeroes are zero.  The pressure term follows transforms of another
order (1e-12 relative L2, as the derivatives); the others are products or copies of
the state's entries, and their transforms run the same passes: equal bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
OM = np.array([0.3, 0.1, -0.2])
_CASES = [("IncompressibleHydro", (16, 24, 32), {"Omega": OM}),
          ("BoussinesqHydro", (32, 16, 16), {"Omega": OM, "beta": 0.4, "boussinesq_direction": "y"}),
          ("BoussinesqHydro", (16, 16, 48), {"beta": -1.5, "boussinesq_direction": "z"})]


def _run(dd, name, shape, params, fused, looks=True):
    M = dd.mods
    p = getattr(M, name)(shape, M.FourierRepresentation)
    p.parameters.update(params)
    if not fused:
        p._advect_fused = lambda data: False
    p._aux_field_list.append(("own", "VectorField"))
    d, o = p.create_fields(0.7), p.create_fields(0.)
    o.add_field("own", "ScalarField")
    rng = np.random.default_rng(8)
    for f, field in d:
        for i, c in field:                  # energy outside the kept modes too
            c["kspace"] = np.transpose(np.fft.rfftn(rng.standard_normal(shape)), (1, 0, 2)) / np.prod(shape)
    assert not hasattr(p, "aux_fields")
    p.RHS(d, o)
    for _ in range(2):                      # further calls, on used work fields if somebody looks at them
        o["own"]["kspace"] = 1.0
        if looks:
            for i, c in p.aux_fields["own"]:
                c["xspace"] = 2.0
            p.aux_fields["mathvector"][0]["xspace"]
        p.RHS(d, o)
    assert not fused or p._advect_fused(d)
    return p, o


@pytest.mark.parametrize("looks", [True, False])
@pytest.mark.parametrize("name,shape,params", _CASES)
def test_work_fields(dd, cuda, name, shape, params, looks):
    (a, oa), (b, ob) = _run(dd, name, shape, params, True, looks), _run(dd, name, shape, params, False)
    assert a.aux_fields is a.aux_fields
    assert a.aux_fields.time == b.aux_fields.time == 0.7
    assert list(a.aux_fields.fields) == list(b.aux_fields.fields)
    for o in (oa, ob):
        assert not np.any(o["own"].to_numpy("kspace"))
    for f, field in b.aux_fields:
        for i, c in field:
            space = c._curr_space                   # as the sequence leaves it
            x, y = a.aux_fields[f][i].to_numpy(space), c.to_numpy(space)
            if f == "mathscalar" and name == "IncompressibleHydro":
                assert np.linalg.norm(x - y) < 1e-12 * np.linalg.norm(y)
            else:
                assert np.array_equal(x, y), (f, i, space)
            assert np.any(y) == (f != "own")


@pytest.mark.parametrize("name,shape,params", _CASES)
def test_derivative_in_the_state_itself(dd, cuda, name, shape, params):
    """RHS(data, data): the sequence zeroes the derivative, so the state, first (physics.py:140-142)."""
    M = dd.mods
    p = getattr(M, name)(shape, M.FourierRepresentation)
    p.parameters.update(params)
    d = p.create_fields(0.7)
    for f, field in d:
        for i, c in field:
            c["xspace"] = np.random.default_rng(i).standard_normal(shape)
    p.RHS(d, d)
    assert not any(np.any(c.to_numpy("kspace")) for f, field in d for i, c in field)
