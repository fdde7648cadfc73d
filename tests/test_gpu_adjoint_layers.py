"""Adjoint windows and column-solver adjoints at layer counts other than the
reference's 26: the sweeps whose depth is a run-time one (up to 64 layers in a
window, 256 in the tracer solver's adjoint).

The bounds are those of the same checks at 26 layers: the window's forward
equals the fused FP64 step to 1e-13 per field, <TL dx, ybar> = <dx, AD ybar>
to 1e-10 (also with a checkpoint stride, whose steps are recomputed), and the
solvers' adjoints agree with central differences to 1e-6."""
import numpy as np
import pytest

import test_gpu_adjoint as dry
import test_gpu_adjoint_moist as moist
import test_gpu_operator_adjoints as operators
from game_archived_gb300 import abi, driver
from helpers import clone, make_model, state_errors
from oracle.bind import Oracle

pytestmark = pytest.mark.gpu

LAYERS = (24, 27, 40, 64)


def _dt(n_layers):
    return 200.0 * min(1.0, 26.0 / n_layers)


def _model(n_layers, is_moist):
    _, m = make_model(3, is_moist, "tracers" if is_moist else "std_wind_tpert", mountain=True, n_layers=n_layers)
    return m


@pytest.mark.parametrize("is_moist", [0, 1], ids=["dry", "moist"])
@pytest.mark.parametrize("n_layers", LAYERS)
def test_window(n_layers, is_moist):
    m, dt = _model(n_layers, is_moist), _dt(n_layers)
    mod = moist if is_moist else dry
    fused = clone(m)
    g = abi.GpuModel(fused, abi.FP64)
    try:
        driver.run(fused, 2, dt, g.linear_combine_two_states, g.manage_rkhevi)
    finally:
        g.close()
    m.config["totally_first_step_bool"][0] = 1
    for stride in (1, 2):
        rng = np.random.default_rng(31 + n_layers)
        out, dy, xb = (mod._state_like(m.layout) for _ in range(3))
        g = abi.GpuModel(m, abi.FP64)
        try:
            g.set_checkpoint_stride(stride)
            g.window_forward(m.state_old, out, dt, 2)
            dx, yb = mod._random_dx(m, rng), mod._random_bar(m, rng)
            g.window_tl(dx, dy)
            g.window_backward(yb, xb)
        finally:
            g.close()
        e = state_errors(out, fused.state_new, m.layout)
        assert max(e.values()) <= 1e-13, e
        lhs, rhs = mod._dot(dy, yb), mod._dot(dx, xb)
        assert abs(lhs - rhs) <= 1e-10 * max(abs(lhs), abs(rhs)), (stride, lhs, rhs)


def _mid_run(n_layers, is_moist):
    m, dt = _model(n_layers, is_moist), _dt(n_layers)
    orc = Oracle(m)
    driver.start(m, orc.linear_combine_two_states)
    for n in range(2):
        driver.step(m, orc.linear_combine_two_states, orc.manage_rkhevi, dt, n * dt)
    return m


@pytest.mark.parametrize("rk", [0, 1])
@pytest.mark.parametrize("n_layers", (27, 64, 65, 100))
def test_tracer_solver(n_layers, rk):
    operators.test_three_band_solver_gen_densities_adj(_mid_run(n_layers, 1), rk)


@pytest.mark.parametrize("rk", [0, 1])
@pytest.mark.parametrize("n_layers", LAYERS)
def test_sound_wave_solver(n_layers, rk):
    operators.test_three_band_solver_ver_waves_adj(_mid_run(n_layers, 0), rk)
