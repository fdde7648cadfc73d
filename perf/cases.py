"""The work a user of this library has it do, as cases that can be timed.

Every case goes through the bindings of the C ABI (game_archived_gb300.abi):

* ``steps``      the reference's time loop (linear_combine_two_states, then
                 manage_rkhevi) on a State the program has on the device, and
                 the copy of the new State to the host at its end;
* ``host``       the same loop in the library's default host-in/host-out mode;
* ``window``     an adjoint window: forward, surface-pressure objective and
                 the gradient with respect to the initial State;
* ``output``     the fields of write_out, on the native and the lat-lon grid;
* ``operators``  single operators on host arrays, as the reference's
                 initialisation and output call them.

The grids are the repository's: RES_ID 3 to 7, 26 layers or another count,
flat or with the 2 km mountain of workloads.py, dry or moist build.  Fields
start from the recipes of cases.py (fewer Lloyd iterations than the benchmark
takes: the cost of a step does not depend on the cells' exact shape), with
noise from the seed.
"""
import ctypes

import numpy as np

from game_archived_gb300 import abi, cases, driver, native, structs, tables, workloads
from game_archived_gb300.ops import CAbiOps

FIELDS = ("rho", "rhotheta_v", "theta_v_pert", "exner_pert", "wind")
DIFFUSION = ("momentum_diff_h", "momentum_diff_v", "temperature_diff_h", "temperature_diff_v", "mass_diff_h",
             "mass_diff_v")
N_LLOYD = {3: 100, 4: 100, 5: 200, 6: 500, 7: 500}
WORK_STRUCTS = ("state_old", "state_new", "state_tendency", "diagnostics", "forcings", "irrev")
N_WIND = 4          # steps of an output interval whose lowest-layer wind enters the 10 m wind


def _case(name, kind, res, layers=26, moist=0, mountain=False, state="std_wind", precision="mixed", steps=1,
          diffusion=False):
    c = dict(kind=kind, res=res, layers=layers, moist=moist, mountain=mountain, state=state, precision=precision,
             steps=steps, diffusion=diffusion)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest grid of the tests and of a first trial run: launches and latency
        _case("steps_r3_mixed_dry", "steps", 3, steps=2),
        # the FP64 parity run with the mountain (RES 5, dry)
        _case("steps_r5_fp64_mountain", "steps", 5, mountain=True, state="std_wind_tpert", precision="fp64", steps=4),
        # the headline workload in FP64
        _case("steps_r6_fp64_moist", "steps", 6, moist=1, state="baroclinic_moist", precision="fp64", steps=2),
        # the headline workload: moist baroclinic jet, mixed precision
        _case("steps_r6_mixed_moist", "steps", 6, moist=1, state="baroclinic_moist", steps=8),
        # the same through the default host-in/host-out calls of a drop-in build
        _case("host_r6_mixed_moist", "host", 6, moist=1, state="baroclinic_moist", steps=2),
        # the largest run: five tracers (clouds everywhere) over the mountain
        _case("steps_r7_mixed_tracers", "steps", 7, moist=1, mountain=True, state="tracers", steps=24),
        # every diffusion switch on, as in the reference's run scripts
        _case("steps_r6_mixed_diffusion", "steps", 6, moist=1, state="baroclinic_moist", steps=12,
              diffusion=True),
        # another layer count than the reference's 26
        _case("steps_r4_mixed_80layers", "steps", 4, layers=80, moist=1, state="jet_moist", steps=4),
        # the adjoint configuration (RES 5, dry, mountain, FP64)
        _case("window_r5_fp64_dry", "window", 5, mountain=True, state="std_wind_tpert", precision="fp64", steps=4),
        # a moist window with the mixed step as the forward of record
        _case("window_r4_mixed_moist", "window", 4, moist=1, mountain=True, state="tracers", steps=3),
        # the output interval of the headline workload
        _case("output_r6_moist", "output", 6, moist=1, state="baroclinic_moist", precision="fp64"),
        # the operators the reference calls outside its time step
        _case("operators_r5", "operators", 5, mountain=True, state="std_wind_tpert", precision="fp64"),
    ]


def draw(rng):
    kind = rng.choice(("steps", "steps", "steps", "steps", "host", "window", "output", "operators"))
    res = rng.choice((3, 4, 4, 5, 5) if kind in ("window", "operators") else (3, 4, 5, 5, 6))
    moist = rng.choice((0, 1, 1))
    mountain = rng.random() < 0.5
    state = rng.choice(("tracers", "jet_moist", "baroclinic_moist") if moist else ("std_wind", "std_wind_tpert"))
    precision = "fp64" if kind in ("output", "operators") else rng.choice(("mixed", "mixed", "fp64"))
    layers = 26
    if kind in ("steps", "host") and rng.random() < 0.4:
        layers = rng.randint(12, 80 if res <= 4 else 40)
    steps = {"steps": rng.randint(1, 12), "host": rng.randint(1, 3), "window": rng.randint(1, 4)}.get(kind, 1)
    if kind == "window" and moist and res == 5:
        steps = min(steps, 2)
    diffusion = kind == "steps" and layers == 26 and rng.random() < 0.3
    return _case(None, kind, res, layers, moist, mountain, state, precision, steps, diffusion)


def _dt(case):
    """the benchmark configurations' time steps: 400 s at RES 4, halved with
    each refinement, and shorter for thinner layers than the 26-layer grid's"""
    return min(400.0, 6400.0 / 2 ** case["res"]) * min(1.0, 26.0 / case["layers"])


# ----------------------------------------------------------- the program
class _Pinned:
    """the library's pinned memory behind one array; given back with the last view of it"""

    def __init__(self, size):
        self.p = ctypes.c_void_p()
        if native.gpu().game_gpu_host_alloc(ctypes.byref(self.p), size) != 0:
            raise abi.GpuError(native.gpu().game_gpu_last_error().decode())

    def __del__(self):
        if self.p.value:
            native.gpu().game_gpu_host_free(self.p)


def pinned(layout, kind="state"):
    """a host struct in the library's pinned memory"""
    size = layout.sizes[kind]
    owner = _Pinned(size)
    mem = (ctypes.c_uint8 * size).from_address(owner.p.value)
    mem.owner = owner
    return structs.HostStruct(layout, kind, np.frombuffer(mem, dtype=np.uint8))


class Program:
    """What a model run holds: the grid, the work structs, the library bound
    to them, and the recipe's initial State.  One at a time, as the library
    has one context per process."""

    now = None

    @staticmethod
    def key(case):
        return tuple(case[k] for k in ("kind", "res", "layers", "moist", "mountain", "state", "precision", "diffusion"))

    @classmethod
    def of(cls, case):
        if cls.now is None or cls.now.k != cls.key(case):
            if cls.now is not None:
                cls.now.gpu.close()
                cls.now = None
            cls.now = cls(case)
        return cls.now

    def __init__(self, case):
        self.k = self.key(case)
        lay = structs.Layout(case["res"], case["layers"], case["moist"])
        self.tab = tables.cached(workloads.input_dir(), case["res"], n_layers=case["layers"],
                                 n_oro_layers=min(23, case["layers"] - 3), n_lloyd=N_LLOYD[case["res"]],
                                 mountain=workloads.MOUNTAIN if case["mountain"] else None)
        m = structs.Model(lay, {k: pinned(lay, "state" if k.startswith("state") else k).buf for k in WORK_STRUCTS})
        self.m = m
        tables.fill_grid(self.tab, m.grid, m.dualgrid)
        cases.default_config(m)
        self.gpu = abi.GpuModel(m, abi.MIXED if case["precision"] == "mixed" else abi.FP64,
                                resident=case["kind"] in ("steps", "output"))
        cases.build_initial_state(m, self.tab, case["state"], CAbiOps(self.gpu.lib, m))
        self.base = m.state_old.clone()
        if case["diffusion"]:
            for s in DIFFUSION:
                m.config[s] = 1
            m.irrev["tke"] = 0.5 + 0.5 * np.random.default_rng(5).random(m.irrev["tke"].size)
        # sedimentation heat, TKE and the diffusion terms carry over from step
        # to step in Irreversible_quantities: a new run gets a fresh struct
        self.irrev = [m.irrev]
        if case["kind"] in ("steps", "host") and (case["state"] == "tracers" or case["diffusion"]):
            self.irrev.append(pinned(lay, "irrev"))
            self.irrev[1].copy_from(m.irrev)

    def initial(self, seed):
        """the recipe's State with the seed's noise on wind, temperature and tracers"""
        lay = self.m.layout
        s, rng = pinned(lay), np.random.default_rng(seed)
        s.copy_from(self.base)
        nc, ne, nl, vpl, ns, gas = lay.nc, lay.ne, lay.nl, lay.vpl, lay.n_scalars, lay.n_cond
        u = s["wind"][:nl * vpl].reshape(nl, vpl)[:, nc:]
        u += rng.standard_normal((nl, ne), dtype=np.float32) * 0.5
        s["theta_v_pert"] += rng.standard_normal(ns, dtype=np.float32) * 0.05
        rho = s["rho"].reshape(lay.n_const, ns)
        s["rhotheta_v"] = rho[gas] * (self.m.grid["theta_v_bg"] + s["theta_v_pert"])
        for k in range(lay.n_const):
            if k != gas:
                rho[k] *= 1.0 + 0.01 * rng.random(ns, dtype=np.float32)
        return s


def prepare(case, seed):
    prog = Program.of(case)
    kind, lay = case["kind"], prog.m.layout
    st = {"case": dict(case), "prog": prog, "init": prog.initial(seed)}
    s = st["init"]
    if kind in ("steps", "output"):
        prog.gpu.sync_to_device(s)
    if kind == "window":
        st["final"], st["bar"], st["grad"] = (pinned(lay) for _ in range(3))
        lat, lon = (prog.m.grid[k][:lay.nc] for k in ("latitude_scalar", "longitude_scalar"))
        p0 = np.radians(45.0)
        inside = np.sin(lat) * np.sin(p0) + np.cos(lat) * np.cos(p0) * np.cos(lon) >= np.cos(np.radians(20.0))
        st["weights"] = np.where(inside, prog.m.grid["area"][lay.n_vectors - lay.nc:lay.n_vectors], 0.0)
    elif kind == "output":
        prog.gpu.record_wind_lowest(s, 0)
        st["buffers"] = prog.gpu.output_fields(s, None, 1, native=True, latlon=True)
    elif kind == "operators":
        st["inputs"] = _operator_inputs(lay, s, seed)
        st["out"] = {"flux": np.zeros(lay.n_vectors), "vort_flux": np.zeros(lay.n_vectors),
                     "kinetic": np.zeros(lay.n_scalars), "gradient": np.zeros(lay.n_vectors),
                     "divergence": np.zeros(lay.n_scalars), "gradient_adj": np.zeros(lay.n_scalars)}
    return st


def run(st):
    case, prog = st["case"], st["prog"]
    gpu, m, init = prog.gpu, prog.m, st["init"]
    kind, dt = case["kind"], _dt(case)
    if kind in ("steps", "host"):
        prog.irrev.reverse()
        m.irrev = prog.irrev[0]
        gpu.linear_combine_two_states(init, init, m.state_new, 1.0, 0.0)
        m.config["totally_first_step_bool"] = 1
        for i in range(case["steps"]):
            driver.step(m, gpu.linear_combine_two_states, gpu.manage_rkhevi, dt, i * dt)
        if kind == "steps":
            gpu.sync_to_host(m.state_new)
        return {f: m.state_new[f] for f in FIELDS}
    if kind == "window":
        m.config["totally_first_step_bool"] = 1
        final, bar, grad = st["final"], st["bar"], st["grad"]
        gpu.window_forward(init, final, dt, case["steps"])
        value = gpu.sfc_pressure_objective(final, st["weights"], bar)
        gpu.window_backward(bar, grad)
        return {"objective": value, "final": {f: final[f] for f in FIELDS}, "gradient": {f: grad[f] for f in FIELDS}}
    if kind == "output":
        for t in range(N_WIND):
            gpu.record_wind_lowest(init, t)
        return gpu.output_fields(init, None, N_WIND, native=True, latlon=True, buffers=st["buffers"])
    i, o = st["inputs"], st["out"]
    gpu.scalar_times_vector(i["density"], i["wind"], o["flux"])
    gpu.calc_pot_vort(i["wind"], i["density"])
    gpu.vorticity_flux(i["mass_flux"], i["pot_vort"], o["vort_flux"])
    gpu.inner_product(i["wind"], i["wind"], o["kinetic"])
    gpu.grad(i["exner"], o["gradient"])
    gpu.divv_h(i["mass_flux"], o["divergence"])
    o["gradient_adj"][:] = 0.0
    gpu.grad_adj(i["mass_flux"], o["gradient_adj"])
    return dict(o, pot_vort=m.diagnostics["pot_vort"], rel_vort=m.diagnostics["rel_vort"])


def _operator_inputs(lay, s, seed):
    rng = np.random.default_rng(seed + 1)
    ns, gas = lay.n_scalars, lay.n_cond
    wind = s["wind"].copy()
    w = wind.reshape(-1)[:lay.nl * lay.vpl].reshape(lay.nl, lay.vpl)[:, :lay.nc]
    w += 0.01 * rng.standard_normal((lay.nl, lay.nc))
    wind[lay.n_vectors - lay.nc:] = 0.0
    return {"density": s["rho"][gas * ns:(gas + 1) * ns].copy(), "wind": wind, "exner": s["exner_pert"].copy(),
            "mass_flux": wind * (0.5 + rng.random(lay.n_vectors)),
            "pot_vort": 1e-8 * (1.0 + rng.random(lay.n_curl))}


# ------------------------------------------------------- what a pass needs
def work(case):
    """Bytes: the State in and out of every step (FP64) and the grid tables
    the operators read, at the precision they are held in; a window reads and
    writes each step's State in both directions, the output pass its fields, an
    operator its arrays.  Operations: counted per point from the reference's
    loops."""
    nl, const = case["layers"], 6 if case["moist"] else 1
    nc = 10 * 4 ** case["res"] + 2
    ne, nt = 3 * (nc - 2), 2 * (nc - 2)
    ns, nv = nl * nc, (nl + 1) * nc + nl * ne
    state = 8 * ((const + 3) * ns + nv)
    wg = 4 if case["precision"] == "mixed" else 8
    grid = wg * (6 * nv + 12 * ns + 16 * ne + 2 * ((nl + 1) * ne + nl * nt)) + 4 * (26 * ne + 12 * nc + 6 * nt)
    flops = ns * (700 + 250 * (const - 1) + (600 if case["diffusion"] else 0))
    n = case["steps"]
    if case["kind"] in ("steps", "host"):
        return {"bytes": n * (2 * state + grid) + state, "flops": n * flops}
    if case["kind"] == "window":
        return {"bytes": n * 2 * (2 * state + grid) + 3 * state, "flops": n * 4 * flops}
    if case["kind"] == "output":
        n_ll = 32768
        fields = 8 * (11 * (nc + n_ll) + 8 * nl * (nc + n_ll) + 7 * 6 * (nc + n_ll) + (nl + 1) * n_ll)
        return {"bytes": state + grid + fields, "flops": ns * 600}
    ncurl = (nl + 1) * ne + nl * ne
    return {"bytes": 8 * (ns + 2 * nv + ns + nv + 2 * ncurl + 2 * nv + ncurl + nv + ns + ns + nv + nv + ns + nv + ns)
            + grid, "flops": ns * 400}


# ------------------------------------------------ 64-bit values, plain numpy
def exact(case, seed):
    """The operators from their definitions; None for the whole step, its
    adjoint and the output pass (a 64-bit run of the whole model)."""
    if case["kind"] != "operators":
        return None
    prog = Program.of(case)
    lay, g = prog.m.layout, prog.m.grid
    nc, ne, nl, vpl = lay.nc, lay.ne, lay.nl, lay.vpl
    i = _operator_inputs(lay, prog.initial(seed), seed)

    def hor(a):                       # [layer][edge] part of a vector field
        return a[:nl * vpl].reshape(nl, vpl)[:, nc:]

    def ver(a):                       # [level][cell] part
        return np.concatenate([a[:nl * vpl].reshape(nl, vpl)[:, :nc], a[nl * vpl:].reshape(1, nc)])

    def vector(h, v):                 # untouched entries stay zero
        a = np.zeros(lay.n_vectors)
        hor(a)[...] = h
        a[:nl * vpl].reshape(nl, vpl)[1:, :nc] = v[1:nl]
        return a

    fr, to = g["from_index"][:ne], g["to_index"][:ne]
    adj = g["adjacent_vector_indices_h"].reshape(nc, 6).copy()
    pent = np.arange(nc) < 12
    adj[pent, 5] = 0
    slot = np.ones((nc, 6))
    slot[pent, 5] = 0.0
    ipw = g["inner_product_weights"].reshape(nl, nc, 8)
    slope, dist, area = (hor(g[k]) for k in ("slope", "normal_distance", "area"))
    dist_v, area_v = ver(g["normal_distance"]), ver(g["area"])
    oro = nl - int(g["no_of_oro_layers"][0])
    rho, ex = i["density"].reshape(nl, nc), i["exner"].reshape(nl, nc)
    wind_h, wind_v = hor(i["wind"]), ver(i["wind"])
    flux_h, flux_v = hor(i["mass_flux"]), ver(i["mass_flux"])
    out = {}
    mid = np.zeros((nl + 1, nc))
    mid[1:nl] = 0.5 * (rho[:-1] + rho[1:]) * wind_v[1:nl]
    out["flux"] = vector(0.5 * (rho[:, fr] + rho[:, to]) * wind_h, mid)
    out["kinetic"] = ((ipw[:, :, :6] * slot * wind_h[:, adj] ** 2).sum(2) + ipw[:, :, 6] * wind_v[:-1] ** 2
                      + ipw[:, :, 7] * wind_v[1:] ** 2).reshape(-1)

    def to_edges(v):                  # a vertical field averaged to the edges of a layer
        c = ipw[:, :, 6] * v[:-1]
        low = ipw[:, :, 7] * v[1:]
        low[-1] = 0.0
        return 0.5 * ((c + low)[:, fr] + (c + low)[:, to])

    grad_v = np.zeros((nl + 1, nc))
    grad_v[1:nl] = (ex[:-1] - ex[1:]) / dist_v[1:nl]
    corr = -slope * to_edges(grad_v)
    corr[:oro] = 0.0
    out["gradient"] = vector((ex[:, to] - ex[:, fr]) / dist + corr, grad_v)
    # divergence with the terrain-following part of the vertical flux
    sign = g["adjacent_signs_h"].reshape(nc, 6) * slot
    tilt = -0.5 * (ipw[:, :, :6] * slot * (slope * flux_h)[:, adj]).sum(2)
    level = np.zeros((nl + 1, nc))
    level[oro] = tilt[oro]
    level[oro + 1:nl] = tilt[oro:nl - 1] + tilt[oro + 1:nl]
    div = (flux_h[:, adj] * sign * area[:, adj]).sum(2) + level[:-1] * area_v[:-1] - level[1:] * area_v[1:]
    out["divergence"] = (div / g["volume"].reshape(nl, nc)).reshape(-1)
    # vorticity flux: the modified TRSK sum and the vertical exchange
    pv = i["pot_vort"]
    pv_h = np.stack([pv[k * 2 * ne:k * 2 * ne + ne] for k in range(nl + 1)])
    pv_v = np.stack([pv[k * 2 * ne + ne:(k + 1) * 2 * ne] for k in range(nl)])
    tw, ti, tm = (g[k].reshape(ne, 10) for k in ("trsk_weights", "trsk_indices", "trsk_modified_curl_indices"))
    total = np.zeros((nl, ne))
    for j in range(10):
        five = (fr if j < 5 else to) < 12
        use = np.where(five, j % 5 < 4, True)
        a, b = np.where(use, ti[:, j], 0), np.where(use, tm[:, j], 0)
        q = pv_v[:, b]
        if j in (2, 7):
            q = np.where(five, q, 0.5 * (q + pv_v))
        total += np.where(use, tw[:, j], 0.0) * flux_h[:, a] * q
    for c in (fr, to):
        total -= 0.5 * ipw[:, c, 6] * flux_v[:-1][:, c] * pv_h[:-1] + 0.5 * ipw[:, c, 7] * flux_v[1:][:, c] * pv_h[1:]
    weight = np.full((nl + 1, 1), 0.5)
    weight[0] = weight[nl] = 1.0
    vert = np.zeros((nl + 1, nc))
    for k in range(nl + 1):
        for layer in (k - 1, k):
            if 0 <= layer < nl:
                vert[k] += (ipw[layer, :, :6] * slot * (flux_h[layer] * pv_h[k])[adj]).sum(1)
    vf = vector(total, weight * vert)
    vf[:nc], vf[nl * vpl:] = (weight * vert)[0], (weight * vert)[nl]
    out["vort_flux"] = vf
    # transpose of the gradient, scattered from its output's bar
    bar_h, bar_v = flux_h, np.zeros((nl + 1, nc))
    bar_v[1:nl] = flux_v[1:nl]
    adj_out = np.zeros((nl, nc))
    for layer in range(nl):
        np.add.at(adj_out[layer], to, bar_h[layer] / dist[layer])
        np.add.at(adj_out[layer], fr, -bar_h[layer] / dist[layer])
        if layer >= oro:
            c = -0.5 * slope[layer] * bar_h[layer]
            for cell in (fr, to):
                np.add.at(bar_v[layer], cell, ipw[layer, cell, 6] * c)
                if layer < nl - 1:
                    np.add.at(bar_v[layer + 1], cell, ipw[layer, cell, 7] * c)
    d = bar_v[1:nl] / dist_v[1:nl]
    adj_out[:-1] += d
    adj_out[1:] -= d
    out["gradient_adj"] = adj_out.reshape(-1)
    return dict(out, pot_vort=None, rel_vort=None)
