"""Constituents that are absent from most of the grid: both paths leave out
their zeros (the FP64 tracer solve writes absent columns, its tendencies skip
zero densities; the mixed path skips layers that hold none of a constituent,
by flags of 32 layers a word).  Snow and cloud water are put into a few layers
of one hemisphere: the FP64 step must match the oracle to 1e-12 of each
constituent's largest value, and the mixed step the FP64 one to 1e-3 of the
largest value in every layer, where a layer left out by mistake would miss its
whole flux divergence.  Layer counts: one word of flags, its edge, two and
three words; both column solvers of the mixed path."""
import numpy as np
import pytest

from game_archived_gb300 import abi, driver
from helpers import clone, make_model, rel_err
from oracle.bind import Oracle

pytestmark = pytest.mark.gpu


def _model(n_layers, layers):
    _, m = make_model(3, 1, "jet_moist", mountain=True, n_layers=n_layers)
    lay = m.layout
    north = m.grid["latitude_scalar"][:lay.nc] > 0.0
    for s in (m.state_old, m.state_new):
        rho = s["rho"].reshape(lay.n_const, n_layers, lay.nc)
        for k, l in enumerate(layers):
            rho[(0, 3)[k % 2], l, north] = 1e-4
    return m


@pytest.mark.parametrize("n_layers,layers,solver", [
    (26, (0, 25), 0), (26, (13, 14), 0), (32, (31, 0), 1), (33, (32, 31), 1), (33, (32, 31), 0), (70, (64, 40), 1)])
def test_absent_constituents(n_layers, layers, solver):
    dt, steps = 150.0 * min(1.0, 26.0 / n_layers), 2
    m64 = _model(n_layers, layers)
    m_orc, m32 = clone(m64), clone(m64)
    for m, precision in ((m64, abi.FP64), (m32, abi.MIXED)):
        g = abi.GpuModel(m, precision, column_solver=solver)
        try:
            driver.run(m, steps, dt, g.linear_combine_two_states, g.manage_rkhevi)
        finally:
            g.close()
    orc = Oracle(m_orc)
    driver.run(m_orc, steps, dt, orc.linear_combine_two_states, orc.manage_rkhevi)
    lay = m64.layout
    shape = (lay.n_const, n_layers, lay.nc)
    r64, r32, ref = (m.state_new["rho"].reshape(shape) for m in (m64, m32, m_orc))
    for k in range(lay.n_const):
        assert rel_err(r64[k], ref[k]) <= 1e-12 * steps, k
        scale = np.abs(r64[k]).max()
        for l in range(n_layers):
            assert np.abs(r32[k, l] - r64[k, l]).max() <= 1e-3 * scale, (k, l)
