"""The pressure-level search of the output pass (GPU) against the oracle where
its FP32 distances cannot decide: a level midway between two layers in ln p, to
within a few units in the last place of FP32 and of FP64, and pressures of
zero, below zero, beyond FP32's range and NaN.

Where both neighbours of a level are equally far, either may count as the
nearest (CUDA's log and the C library's differ in the last bits).  The
interpolation is then the same but for the 1e-10 that keeps its denominator,
0.2 here, from zero: the weights differ by 1e-10 / 0.2 / 2 = 2.5e-10, the fields
by no more than twice that of their largest magnitude."""
import numpy as np
import pytest

from game_archived_gb300 import abi
from helpers import clone, output_scenario
from oracle import bind

pytestmark = pytest.mark.gpu

TOL = 5e-10 + 1e-11  # and the bound of the output fields
R_D = 287.057811  # only places the pressures: the oracle and the library get the same densities


@pytest.mark.parametrize("level", [0, 2, 5])
def test_pressure_levels_where_fp32_cannot_decide(level):
    pl = (20000., 30000., 50000., 70000., 85000., 92500.)[level]
    m, wl, nw = output_scenario(3, 0, "std_wind_tpert", False)
    lay = m.layout
    nc, nl = lay.nc, lay.nl
    m_t = clone(m)
    orc = bind.Oracle(m_t)
    bind.write_out_fields(orc, m_t.state_new, wl, nw)
    t = m_t.diagnostics["temperature"].reshape(nl, nc)
    rho = m.state_new["rho"][:nl * nc].reshape(nl, nc)
    p = rho * R_D * t
    upper = np.clip(np.argmin(np.abs(np.log(p / pl)), axis=0), 1, nl - 2)
    cols = np.arange(0, nc, 3)
    for n, c in enumerate(cols):
        k = upper[c]
        off = (0.0, 1e-16, -1e-15, 1e-12, 1e-7, -3e-7, 9e-4, -1.1e-3)[n % 8]
        rho[k, c] = pl * np.exp(-0.1 + off) / (R_D * t[k, c])
        rho[k + 1, c] = pl * np.exp(0.1) / (R_D * t[k + 1, c])
    for n, c in enumerate(np.arange(1, nc, 3)):
        rho[n % nl, c] = (0.0, -1.0, 1e36, np.nan, 1e-36, np.inf)[n % 6]
    m_o = clone(m)
    with np.errstate(all="ignore"):
        ref = bind.write_out_fields(bind.Oracle(m_o), m_o.state_new, wl, nw)
    g = abi.GpuModel(m, abi.FP64)
    try:
        got = g.output_fields(m.state_new, wl, nw, native=True)["native"]
    finally:
        g.close()
    for name in ("geopotential_height", "t_pl", "u_pl", "v_pl"):
        a, b = got[name], ref[name]
        assert np.array_equal(a == 9999, b == 9999), name
        assert np.array_equal(np.isnan(a), np.isnan(b)), name
        ok = np.isfinite(b) & (b != 9999)
        assert np.max(np.abs(a[ok] - b[ok])) <= TOL * np.max(np.abs(b[ok])), name
