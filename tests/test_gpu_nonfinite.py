"""Single operators on fields that hold infinities and NaN: the values they
come from and go to are the oracle's, on flat grids (slopes and height
differences of exactly 0, whose products are NaN then) and with a mountain.
Finite results to 1e-12 of the largest as in the operators' other tests."""
import numpy as np
import pytest

from game_archived_gb300 import abi
from helpers import make_model
from oracle.bind import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(1, True), (0, False)], ids=["moist-mountain", "dry-flat"])
def setup(request):
    moist, mountain = request.param
    _, m = make_model(3, moist, "tracers" if moist else "std_wind", mountain)
    g = abi.GpuModel(m, abi.FP64)
    yield m, g, Oracle(m)
    g.close()


def _same(a, b):
    """the same infinities and NaN in the same places, finite values close"""
    for f in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(f(a), f(b)), (f.__name__, np.flatnonzero(f(a) != f(b))[:10])
    ok = np.isfinite(b)
    assert not ok.all()
    assert np.abs(a[ok] - b[ok]).max() <= 1e-12 * np.abs(b[ok]).max()


def _spoil(m, field, stride, lead):
    """+inf, -inf and NaN in the top layer, in the middle and in the lowest"""
    lay = m.layout
    for layer, where, value in ((0, 40, np.inf), (12, 100, -np.inf), (lay.nl - 1, 300, np.nan), (20, 500, np.inf)):
        field[layer * stride + lead + where] = value


def test_grad(setup):
    m, g, o = setup
    lay = m.layout
    f = m.state_old["exner_pert"].copy()
    _spoil(m, f, lay.nc, 0)
    a, b = np.zeros(lay.n_vectors), np.zeros(lay.n_vectors)
    g.grad(f, a)
    o.grad(f, b)
    _same(a, b)


def test_calc_pot_vort(setup):
    m, g, o = setup
    lay, d = m.layout, m.diagnostics
    rho = m.state_old["rho"][lay.n_cond * lay.n_scalars:(lay.n_cond + 1) * lay.n_scalars].copy()
    for lead in (0, lay.nc):            # vertical, horizontal wind
        wind = m.state_old["wind"].copy()
        _spoil(m, wind, lay.vpl, lead)
        got = {}
        g.calc_pot_vort(wind, rho)
        for k in ("rel_vort_on_triangles", "rel_vort", "pot_vort"):
            got[k] = d[k].copy()
        o.calc_pot_vort(wind, rho)
        for k in got:
            if lead or k != "rel_vort_on_triangles":
                _same(got[k], d[k])


def test_pressure_gradient(setup):
    m, g, o = setup
    s = m.state_old.clone()
    _spoil(m, s["exner_pert"], m.layout.nc, 0)
    g.manage_pressure_gradient(s)
    got = m.forcings["pressure_gradient_acc_neg_nl"].copy()
    o.manage_pressure_gradient(s)
    _same(got, m.forcings["pressure_gradient_acc_neg_nl"])


def test_state_copy_is_the_linear_combination(setup):
    """coefficients 1 and 0, the time loop's copy: 1 a + 0 b bit for bit, signed
    zeros, infinities and NaN of either State included"""
    m, g, _ = setup
    v = np.array([0.0, -0.0, 1.5, -2.5, np.inf, -np.inf, np.nan, 5e-324, -5e-324])
    a, b, out = m.state_old.clone(), m.state_old.clone(), m.state_old.clone()
    for f in ("rho", "rhotheta_v", "exner_pert", "wind"):
        n = a[f].size
        a[f][:] = np.resize(np.repeat(v, v.size), n)
        b[f][:] = np.resize(np.tile(v, v.size), n)
    g.linear_combine_two_states(a, b, out, 1.0, 0.0)
    for f in ("rho", "rhotheta_v", "exner_pert", "wind"):
        with np.errstate(all="ignore"):
            want = 1.0 * a[f] + 0.0 * b[f]
        same = (out[f].view(np.uint64) == want.view(np.uint64)) | (np.isnan(out[f]) & np.isnan(want))
        assert same.all(), (f, a[f][~same][:5], b[f][~same][:5], out[f][~same][:5])
