"""The mixed path's flags of the layers that hold a constituent: leaving a layer
out must not change a bit.

Condensates are put into every other cell of a hemisphere in a few layers; the
same run is made with a trace (1e-30) of every condensate in every layer of one
far cell, which sets every flag.  Away from that cell the two must agree to the
bit: a layer wrongly left out would miss the whole flux of its constituent.
That there is such a flux, and that layers are left out, is asserted.  Layer
counts of one word of flags, its edge, two and three words; flat and with a
mountain (columns with and without the terrain terms); both column solvers and
both arithmetics of the eliminations; and with the diffusion branch, whose
scalar fluxes go by the same flags."""
import numpy as np
import pytest

from game_archived_gb300 import abi, driver
from helpers import make_model

pytestmark = pytest.mark.gpu

SWITCHES = ("momentum_diff_h", "momentum_diff_v", "temperature_diff_h", "temperature_diff_v", "mass_diff_h",
            "mass_diff_v")
STEPS = 2


def _run(n_layers, layers, mountain, solver, dfloat, diffusion, traced):
    _, m = make_model(3, 1, "jet_moist", mountain=mountain, n_layers=n_layers)
    lay = m.layout
    lat = m.grid["latitude_scalar"][:lay.nc]
    cells = np.flatnonzero((lat > 0.0) & (np.arange(lay.nc) % 2 == 0))
    shape = (lay.n_const, n_layers, lay.nc)
    for k, l in enumerate(layers):
        m.state_old["rho"].reshape(shape)[(0, 3)[k % 2], l, cells] = 1e-4
    if diffusion:
        for s in SWITCHES:
            m.config[s] = 1
        m.irrev["tke"][:] = 0.5 + 0.5 * np.random.default_rng(5).random(m.irrev["tke"].size)
    start = m.state_old["rho"].reshape(shape).copy()
    far = int(np.argmin(lat))
    dt = 150.0 * min(1.0, 26.0 / n_layers)
    g = abi.GpuModel(m, abi.MIXED, column_solver=solver, double_float=dfloat)
    try:
        driver.start(m, g.linear_combine_two_states)
        for i in range(STEPS):
            if traced:
                rho = m.state_new["rho"].reshape(shape)
                rho[:lay.n_cond, :, far] = np.maximum(rho[:lay.n_cond, :, far], 1e-30)
            driver.step(m, g.linear_combine_two_states, g.manage_rkhevi, dt, i * dt)
    finally:
        g.close()
    xyz = np.stack([np.cos(lat) * np.cos(lon := m.grid["longitude_scalar"][:lay.nc]), np.cos(lat) * np.sin(lon),
                    np.sin(lat)])
    apart = xyz.T @ xyz[:, far] < np.cos(1.0)
    return start, {f: m.state_new[f].copy() for f in ("rho", "rhotheta_v", "theta_v_pert", "exner_pert")}, apart


@pytest.mark.parametrize("n_layers,layers,mountain,solver,dfloat,diffusion", [
    (26, (0, 25), True, 0, 1, False), (26, (13, 14), False, 0, 1, False), (26, (13, 14), True, 0, 0, False),
    (26, (5, 24), True, 0, 1, True), (26, (5, 24), False, 0, 1, True),
    (32, (31, 0), False, 1, 1, False), (33, (32, 31), False, 1, 1, False), (33, (32, 31), True, 2, 1, False),
    (33, (32, 31), False, 0, 1, False), (64, (63, 32), False, 1, 1, False), (65, (64, 63), False, 1, 1, False),
    (70, (64, 40), True, 1, 1, False), (70, (64, 40), False, 2, 1, False)])
def test_left_out_layers_change_nothing(n_layers, layers, mountain, solver, dfloat, diffusion):
    start, a, apart = _run(n_layers, layers, mountain, solver, dfloat, diffusion, False)
    _, b, _ = _run(n_layers, layers, mountain, solver, dfloat, diffusion, True)
    rho = a["rho"].reshape(start.shape)
    for k, l in enumerate(layers):      # carried to cells that held none
        c = (0, 3)[k % 2]
        assert ((start[c, l] == 0.0) & (rho[c, l] > 0.0) & apart).sum() > 50, (c, l)
    assert (rho == 0.0).all(axis=2).any()               # a constituent absent from a layer at the end
    assert (start[:4] == 0.0).all(axis=2).sum() >= 4 * n_layers - 4
    for f in a:
        x, y = (v[f].reshape(-1, apart.size)[:, apart] for v in (a, b))
        bad = np.argwhere(x != y)
        assert bad.size == 0, (f, len(bad), bad[:5], x[tuple(bad[0])], y[tuple(bad[0])])
