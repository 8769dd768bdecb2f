"""Operators, representations and k^2 that a user's program replaces are used by the
3D rotating and Boussinesq right-hand sides at every size: the one-call path
(dd_advect_rhs3d) stands aside for them.  The expected result is the operator
sequence itself, so outputs are equal bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SHAPE = (16, 24, 16)
PARAMS = {"IncompressibleHydro": {"Omega": np.array([0.3, 0.1, -0.2])},
          "BoussinesqHydro": {"Omega": np.array([0.3, 0.1, -0.2]), "g": 1.3, "boussinesq_direction": "y"}}


def _rhs(phys, k, patch=None):
    """Right-hand side of the state k (field, component) as numpy arrays, with _advect_fused replaced by patch."""
    if patch is not None:
        phys._advect_fused = patch
    d, o = phys.create_fields(0.), phys.create_fields(0.)
    for f, field in d:
        for i, c in field:
            c["kspace"] = k[f, i]
    phys.RHS(d, o)
    return [c.to_numpy("kspace") for f, field in o for i, c in field]


def _make(dd, base, rep=None, **over):
    M = dd.mods
    cls = type("Own" + base, (getattr(M, base),), over)
    phys = cls(SHAPE, rep or M.FourierRepresentation)
    phys.parameters.update(PARAMS[base])
    return phys


def _state():
    rng = np.random.default_rng(3)
    return {(f, i): np.transpose(np.fft.rfftn(rng.standard_normal(SHAPE)), (1, 0, 2)) / np.prod(SHAPE)
            for f, n in (("u", 3), ("T", 1)) for i in range(n)}


def _check(stock, own):
    """own() makes the changed physics; its results are those of its operator sequence, and not the stock ones."""
    k = _state()
    a, b, s = _rhs(own(), k), _rhs(own(), k, lambda data: False), _rhs(stock, k)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
    assert any(np.linalg.norm(x - y) > 1e-3 * np.linalg.norm(y) for x, y in zip(a, s))


def _scaled(name, out):
    """Operator `name` of the stock class with its output (argument out) doubled afterwards."""
    def method(self, *args):
        getattr(super(type(self), self), name)(*args)
        for i, c in args[out]:
            c["kspace"] = 2 * c["kspace"]
    return method


@pytest.mark.parametrize("base", list(PARAMS))
@pytest.mark.parametrize("name,out", [("XgradY", 4), ("divX", 1), ("XconstcrossY", 2), ("laplace_solve", 1)])
def test_operators_of_a_subclass(dd, cuda, base, name, out):
    _check(_make(dd, base), lambda: _make(dd, base, **{name: _scaled(name, out)}))


@pytest.mark.parametrize("base", list(PARAMS))
def test_no_projection(dd, cuda, base):
    _check(_make(dd, base), lambda: _make(dd, base, pressure_projection=lambda self, data, deriv: None))


def test_operator_of_an_instance(dd, cuda):
    def own():
        p = _make(dd, "BoussinesqHydro")
        p.pressure_projection = lambda data, deriv: None
        return p
    _check(_make(dd, "BoussinesqHydro"), own)


@pytest.mark.parametrize("base", list(PARAMS))
def test_representation(dd, cuda, base):
    F = dd.mods.FourierRepresentation

    class Damped(F):
        def deriv(self, dim):
            d = F.deriv(self, dim)
            d *= 0.5
            return d
    _check(_make(dd, base), lambda: _make(dd, base, rep=Damped))


@pytest.mark.parametrize("base", list(PARAMS))
def test_k2_of_the_user(dd, cuda, base):
    def own():
        p = _make(dd, base)
        p.k2 = p.create_fields(0.)["u"][0].k2(no_zero=True) + 3.0
        return p
    _check(_make(dd, base), own)


@pytest.mark.parametrize("base", list(PARAMS))
def test_stock_classes_take_one_call(dd, cuda, base):
    """A subclass that changes nothing, and the classes themselves, keep the one-call path."""
    for p in (_make(dd, base), _make(dd, base, own_attribute=1)):
        d, o = p.create_fields(0.), p.create_fields(0.)
        p.RHS(d, o)
        assert p._advect_fused(d)
        p.RHS(d, o)
        assert p._advect_fused(d)


@pytest.mark.parametrize("base", list(PARAMS))
def test_k2_after_a_right_hand_side(dd, cuda, base):
    """The k^2 that laplace_solve caches at the first call is there, reading it changes nothing, and
    writing to it, in place or not, reaches the pressure solve."""
    p, s = _make(dd, base), _make(dd, base)
    s._advect_fused = lambda data: False
    assert p.k2 is None and s.k2 is None
    k = _state()
    first = _rhs(p, k)
    _rhs(s, k)
    assert np.array_equal(p.k2.cpu().numpy(), s.k2.cpu().numpy()) and p.k2 is p.k2
    assert p._advect_fused(p.create_fields(0.))
    assert all(np.array_equal(x, y) for x, y in zip(_rhs(p, k), first))
    for change in (lambda q: q.k2.add_(3.0), lambda q: setattr(q, "k2", q.k2 * 2.0)):
        change(p)
        change(s)
        assert all(np.array_equal(x, y) for x, y in zip(_rhs(p, k), _rhs(s, k)))
    p = _make(dd, base)
    p.laplace_k2 = "current"
    _rhs(p, k)
    assert p.k2 is None
