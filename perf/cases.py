"""The work that users of athad_cond_b200 have it do, as cases that can be timed and compared.

Every case starts from the model's own initial state (GpuAtmosphere.initial_state) of a
condition point that the seed draws (40-100 bar, sea surface 503-523 K, the ensemble's
ranges), with a seeded Gaussian velocity perturbation: the states that the model steps
through in earnest, other ones for every seed.  Outputs are views of the context's device
fields, so a pass copies nothing to the host that a program would not read.

Kinds: "rk4" one time step; "project" the initial projection of the velocities; "solve" the
pressure equation to a tolerance; "satadj", "moist", "ice", "radiation" one physics module;
"loop" four whole model iterations (the cadence's period); "ensemble" four iterations of a
batch of members.
"""
import math

import numpy as np
import torch

from athad_cond_b200 import GpuAtmosphere, GpuBatch
from athad_cond_b200.ensemble import condition_params, draw_condition, draw_ensemble, init_config
from athad_cond_b200._abi import Precision
from athad_cond_b200.loop import CONVECTION_FIELDS, ModelLoop, TURBULENCE_FIELDS

DT = 4e-5
Y = ("t", "u", "v", "w", "c", "cloud", "ice", "gr", "co2", "tke", "dis")
AUX = ("aux_u", "aux_v", "aux_w")
SOURCES = ("S_v", "S_c", "S_i", "S_r", "S_s")
SPIN_UP = 5        # iterations before a moist module's case: the next iteration is a moist one


def listed():
    return [
        # the reference's own grid in its own precision, the turbulence closure it configures
        {"name": "rk4_fp64_61x181x361", "kind": "rk4", "im": 61, "jm": 181, "km": 361, "precision": "fp64",
         "turb": 3, "diag": 0},
        # the benchmark's grid and form
        {"name": "rk4_mixed_41x181x361", "kind": "rk4", "im": 41, "jm": 181, "km": 361, "precision": "mixed",
         "turb": 3, "diag": 0},
        # a ragged grid as ensembles draw them, k-epsilon, with the step's diagnostic outputs
        {"name": "rk4_mixed_27x117x245", "kind": "rk4", "im": 27, "jm": 117, "km": 245, "precision": "mixed",
         "turb": 1, "diag": 1},
        # every run starts with 200 sweeps of the initial projection: a chain of small launches
        {"name": "project_41x181x361", "kind": "project", "im": 41, "jm": 181, "km": 361, "sweeps": 200},
        # the pressure-Poisson stress solve, the largest grid of the benchmark
        {"name": "solve_61x361x721", "kind": "solve", "im": 61, "jm": 361, "km": 721},
        # the moist iteration's column modules on the state they meet at a moist iteration
        {"name": "satadj_41x181x361", "kind": "satadj", "im": 41, "jm": 181, "km": 361},
        {"name": "moist_41x181x361", "kind": "moist", "im": 41, "jm": 181, "km": 361},
        {"name": "ice_41x181x361", "kind": "ice", "im": 41, "jm": 181, "km": 361, "category": 2},
        # radiation runs every iteration
        {"name": "radiation_61x181x361", "kind": "radiation", "im": 61, "jm": 181, "km": 361},
        # the whole model: the benchmark's grid, and a serving grid where launches and host work count
        {"name": "loop_mixed_41x181x361", "kind": "loop", "im": 41, "jm": 181, "km": 361, "precision": "mixed"},
        {"name": "loop_fp64_21x91x181", "kind": "loop", "im": 21, "jm": 91, "km": 181, "precision": "fp64"},
        # many members of uneven grids advanced together
        {"name": "ensemble_6", "kind": "ensemble", "members": 6, "grids": 20261203},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(n):
    return n | 1


def draw(rng):
    kind = rng.choice(("rk4", "rk4", "project", "solve", "satadj", "moist", "ice", "radiation", "loop", "ensemble"))
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(2, 6), "grids": rng.randrange(1 << 30)}
    big = kind == "solve"      # the solve alone is used on grids beyond the model's own
    c = {"kind": kind, "im": rng.randint(11, 61), "jm": _odd(_log_int(rng, 21, 350 if big else 180)),
         "km": _odd(_log_int(rng, 41, 700 if big else 360))}
    if kind == "rk4":
        c.update(precision=rng.choice(("fp64", "mixed")), turb=rng.randint(1, 3), diag=rng.randint(0, 1))
    elif kind == "project":
        c.update(sweeps=_log_int(rng, 2, 200))
    elif kind == "ice":
        c.update(category=rng.randint(0, 3) if c["im"] >= 24 else 2)
    elif kind == "loop":
        c.update(precision=rng.choice(("fp64", "mixed")))
    return c


class _Field:
    """A context's device field as an array that torch reads in place; it keeps the context."""

    def __init__(self, g, name):
        self.g = g
        im, jm, km = g.shape
        ptr, pitch = g.device_ptr(name)
        self.__cuda_array_interface__ = {"shape": (im, jm, km), "strides": (jm * pitch * 8, pitch * 8, 8),
                                         "typestr": "<f8", "data": (ptr, False), "version": 3}


def _views(g, names):
    return {n: torch.as_tensor(_Field(g, n), device="cuda") for n in names}


_stream = None


def _program_stream():
    """The one stream that a program gives to its contexts."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


def _context(case, seed):
    """A context in its initial state at the seed's condition point, the velocities perturbed."""
    cond = draw_condition(np.random.default_rng(seed))
    p = condition_params(cond, Precision.MIXED if case.get("precision") == "mixed" else Precision.FP64)
    p.turb_model = case.get("turb", p.turb_model)
    p.category_ice_scheme = case.get("category", p.category_ice_scheme)
    g = GpuAtmosphere(case["im"], case["jm"], case["km"], p)
    g.set_stream(_program_stream())
    g.initial_state(init_config(cond))
    g.synchronize()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for x in _views(g, ("u", "v", "w")).values():
        # 0.05 m/s in the model's unit of 8 m/s
        x[1:-1, 1:-1, 1:-1] += (0.05 / 8.0) * torch.randn(x[1:-1, 1:-1, 1:-1].shape, generator=gen,
                                                        dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    g.storeIntermediateData3D()
    g.synchronize()
    return g


def _outputs(kind, case):
    """Names of the fields that a pass computes."""
    if kind == "rk4":
        names = Y + AUX
        return names + (("prod", "tke_source", "dis_source", "CoriolisForce", "BuoyancyForce",
                         "PressureGradientForce") if case["diag"] else tuple(n + "n" for n in Y))
    return {"project": ("u", "v", "w"), "solve": ("p_dyn",),
            "satadj": ("t", "c", "cloud", "ice", "S_c_c"),
            "moist": CONVECTION_FIELDS + ("MC_q", "u_u", "v_u", "w_u", "u_d", "v_d", "w_d", "D_u", "D_d",
                                         "p_stat", "r_humid", "r_dry", "co2"),
            "ice": ("c", "cloud", "ice", "P_rain", "P_snow") + SOURCES,
            "radiation": ("t", "radiation", "epsilon"),
            "loop": Y + TURBULENCE_FIELDS[2:] + ("p_dyn", "p_stat", "r_humid", "P_rain", "P_snow", "P_conv",
                                                 "Precipitation", "MC_t", "MC_v", "MC_w", "TempDewPoint",
                                                 "HumidityRel", "radiation", "Q_Sensible"),
            "ensemble": ("t", "u", "v", "w", "c", "cloud", "co2", "tke", "p_dyn", "r_humid")}[kind]


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "kind": kind}
    if kind == "ensemble":
        rng = np.random.default_rng(seed)
        members = []
        for m in draw_ensemble(case["members"], case["grids"]):
            members.append(_context({"im": m.grid[0], "jm": m.grid[1], "km": m.grid[2], "precision": "mixed"},
                                    int(rng.integers(1 << 30))))
        state["batch"] = GpuBatch(members, dt=DT)
        state["batch"].set_stream(_program_stream())
        state["out"] = [_views(g, _outputs(kind, case)) for g in members]
        return state
    g = state["g"] = _context(case, seed)
    if kind == "loop":
        state["loop"] = ModelLoop(g, dt=DT)
    elif kind in ("satadj", "moist", "ice"):
        ModelLoop(g, dt=DT).run(SPIN_UP)
    if kind == "solve":
        # the stress source: a 0.5 m/s Gaussian velocity perturbation
        gen = torch.Generator(device="cuda").manual_seed(seed)
        for n in AUX:
            x = (0.5 / 8.0) * torch.randn(g.shape, generator=gen, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            g.upload_tensor(n, x)
            g.synchronize()
    if kind == "moist":
        g.SaturationAdjustment_run()
    if kind == "satadj":
        # what the transport hands over; the adjustment works in place, so a pass takes it anew
        g.synchronize()
        state["given"] = {n: x.contiguous() for n, x in _views(g, ("t", "c", "cloud", "ice")).items()}
    state["out"] = _views(g, _outputs(kind, case))
    g.synchronize()
    return state


def run(state):
    kind, case, g = state["kind"], state["case"], state.get("g")
    if kind == "rk4":
        # with diagnostics as the whole model calls it, otherwise as the benchmark does
        g.solveRungeKutta_Atmosphere_Turb(DT, 1.0, 0.01, write_diagnostics=case["diag"],
                                          store_n_level=not case["diag"])
    elif kind == "project":
        g.project_initial_velocity(case["sweeps"])
    elif kind == "solve":
        g.fill("p_dyn", 0.0)
        g.pressure_solve(1e-10, 500)
    elif kind == "satadj":
        for n, x in state["given"].items():
            g.upload_tensor(n, x)
        g.SaturationAdjustment_run()
    elif kind == "moist":
        g.MoistConvection_run(SPIN_UP + 1)
        g.densities()
    elif kind == "ice":
        g.ice_scheme()
    elif kind == "radiation":
        g.radiative_heating(0.05)
    elif kind == "loop":
        said = state["loop"].run(4)
        return {"fields": state["out"], "t_skin": [r["t_skin"] for r in said],
                "residuum": [r["residuum"]["residuum"] for r in said],
                "water": [r["h2o"]["q_mean"] for r in said if "h2o" in r],
                "co2": [r["co2"]["q_mean"] for r in said if "co2" in r]}
    elif kind == "ensemble":
        for _ in range(4):
            state["batch"].iteration(graph=True)
    return state["out"]


# Fields read and written once per pass and cell, FP64 (the entry points' own fields), and
# floating-point operations per cell.
_FIELDS = {"project": 6, "solve": 5, "satadj": 4 + 7 + 5, "moist": 14 + 31 + 9, "ice": 12 + 11, "radiation": 6 + 3,
           "loop": 4 * (37 + 25 + 9) + 2 * 120}
_FLOPS = {"satadj": 1500, "moist": 1500, "ice": 800, "radiation": 300, "loop": 4 * 3500 + 2 * 5000}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        n = sum(a * b * c for a, b, c in (m.grid for m in draw_ensemble(case["members"], case["grids"])))
        return {"bytes": 8.0 * n * (4 * 62 + 2 * 70), "flops": 1.0 * n * (4 * 2800 + 2 * 3000)}
    n = case["im"] * case["jm"] * case["km"]
    if kind == "rk4":      # 11 state, 11 time level n, 15 forcing in; 11 state, 3 forces, diagnostics or level n out
        return {"bytes": 8.0 * n * (37 + 14 + (8 if case["diag"] else 11)), "flops": 2800.0 * n}
    if kind == "project":
        return {"bytes": 8.0 * n * _FIELDS[kind], "flops": n * (15.0 * case["sweeps"] + 30.0)}
    if kind == "solve":    # about thirty preconditioned iterations
        return {"bytes": 8.0 * n * _FIELDS[kind], "flops": 30.0 * 150.0 * n}
    return {"bytes": 8.0 * n * _FIELDS[kind], "flops": 1.0 * n * _FLOPS[kind]}


# ---- the same results in 64 bits from plain torch --------------------------------------
# For the column modules with data-dependent iterations and branches (the saturation
# adjustment, the convection, the ice schemes) and for whole iterations there is none: a
# second text of the whole scheme would be needed, and the solve's would take minutes.


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "rk4":
            return _exact_rk4(case, seed)
        if case["kind"] == "project":
            return _exact_project(case, seed)
        if case["kind"] == "radiation":
            return _exact_radiation(case, seed)
    return None


class _Grid:
    """The model's metric factors (spherical shell, exponentially stretched radius)."""

    def __init__(self, g):
        p, (im, jm, km) = g.params, g.shape
        f = dict(dtype=torch.float64, device="cuda")
        self.dr, self.dthe, self.dphi = 1.0 / (im - 1), math.pi / (jm - 1), 2.0 * math.pi / (km - 1)
        rad = 1.0 + self.dr * torch.arange(im, **f)
        the = self.dthe * torch.arange(jm, **f)
        self.shell = (math.exp(p.zeta) - 1.0) * p.L_atm
        r0 = p.r_Earth * 1e3 / self.shell if p.metric_r0 < 0 else p.metric_r0
        rmet = (r0 + (rad - 1.0) if r0 > 0 else rad)[:, None, None]
        self.exp = (1.0 / (rad + 1.0))[:, None, None]
        self.sin_w = torch.sin(the)
        self.sin = self.sin_w.clamp(min=0.55)[None, :, None]
        self.cos = torch.cos(the)[None, :, None]
        self.ir, self.irs = 1.0 / rmet, 1.0 / (rmet * self.sin)
        self.height = torch.tensor([float(np.float32((math.exp(p.zeta * i * self.dr) - 1) * float(np.float32(p.L_atm))))
                                    for i in range(im)], **f)


def _fields(g, names):
    g.synchronize()
    return {n: x.clone() for n, x in _views(g, names).items()}


def _star(x):
    c = x[1:-1, 1:-1, 1:-1]
    return (c, x[2:, 1:-1, 1:-1], x[:-2, 1:-1, 1:-1], x[1:-1, 2:, 1:-1], x[1:-1, :-2, 1:-1],
            x[1:-1, 1:-1, 2:], x[1:-1, 1:-1, :-2])


def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _exact_rk4(case, seed):
    g = _context(case, seed)
    p, m = g.params, _Grid(g)
    f = _fields(g, Y + tuple(n + "n" for n in Y) + SOURCES + (
        "S_g", "p_dyn", "nue", "t_eq", "p_stat", "r_humid", "MC_t", "MC_q", "MC_v", "MC_w"))
    I = (slice(1, -1),) * 3
    inner = (slice(1, -1),)
    ex, ir, irs = m.exp[inner], m.ir[inner], m.irs[:, 1:-1][inner]
    sn, cs = m.sin[:, 1:-1], m.cos[:, 1:-1]
    im, jm, km = g.shape
    w = m.sin_w[None, :, None]
    t_ref = (f["t"] * w).sum((1, 2), keepdim=True)[inner] / (m.sin_w.sum() * km)
    inv_re = 1.0 / p.re_turb
    force = p.omega * m.shell / p.u_0
    nue, rh = f["nue"][I], f["r_humid"][I]
    ce = 1.0 / (p.c_0 * p.cp_l * p.t_0)
    sigma = torch.where(f["p_stat"][:1] > 0, f["p_stat"] / f["p_stat"][:1], torch.zeros_like(f["p_stat"]))[I]
    k_a, k_s = 1 / (4 * 86400.0), 1 / (0.4 * 86400.0)
    k_T = (k_a + (k_s - k_a) * ((sigma - 0.7) / 0.3).clamp(min=0) * sn ** 4) * p.L_atm / p.u_0
    source = {"t": p.L_atm / (p.u_0 * p.t_0) * f["MC_t"][I]
              + ce * rh * (p.lv * (f["S_c"] + f["S_r"])[I] + p.ls * (f["S_i"] + f["S_s"] + f["S_g"])[I]),
              "c": f["S_v"][I] * rh + p.L_atm / (p.u_0 * p.c_0) * f["MC_q"][I], "cloud": f["S_c"][I] * rh,
              "ice": f["S_i"][I] * rh, "gr": f["S_g"][I] * rh, "co2": 0.0}
    dp = {}
    _, a, b, c_, d, e, h = _star(f["p_dyn"])
    dp["r"], dp["t"], dp["p"] = (a - b) / (2 * m.dr), (c_ - d) / (2 * m.dthe), (e - h) / (2 * m.dphi)
    drag = (1.0 - torch.arange(1, im - 1, dtype=torch.float64, device="cuda")[:, None, None] / 5.0).clamp(0, 1)
    drag = drag * (p.L_atm / p.u_0 * DT / 86400.0)
    ar = [torch.arange(1, n - 1, dtype=torch.float64, device="cuda") for n in (im, jm, km)]
    dj = torch.minimum(ar[1], jm - 1 - ar[1]) if p.wall_mode == 0 else ar[1]
    wall = torch.minimum(torch.minimum(ar[0][:, None, None], dj[None, :, None]), ar[2][None, None, :])
    MCV = p.L_atm / (p.u_0 * p.u_0)

    def rhs(y):
        s = {n: _star(y[n]) for n in Y}
        d1 = {n: ((x[1] - x[2]) / (2 * m.dr), (x[3] - x[4]) / (2 * m.dthe), (x[5] - x[6]) / (2 * m.dphi))
              for n, x in s.items()}
        U, V, W = s["u"][0], s["v"][0], s["w"][0]
        ur, vt, wp = U * ex, V * ir, W * irs

        def second(n):
            x = s[n]
            return ((x[1] - 2 * x[0] + x[2]) / m.dr ** 2 * ex ** 2, (x[3] - 2 * x[0] + x[4]) / m.dthe ** 2 * ir ** 2,
                    (x[5] - 2 * x[0] + x[6]) / m.dphi ** 2 * irs ** 2)

        def laplace(n):
            return sum(second(n)) + d1[n][0] * 2 * ir * ex + d1[n][1] * cs / sn * ir ** 2

        def limited(n):
            x = s[n]
            return (ur * _minmod(x[0] - x[2], x[1] - x[0]) / m.dr + vt * _minmod(x[0] - x[4], x[3] - x[0]) / m.dthe
                    + wp * _minmod(x[0] - x[6], x[5] - x[0]) / m.dphi)

        def central(n):
            return ur * d1[n][0] + vt * d1[n][1] + wp * d1[n][2]

        k, om = s["tke"][0], s["dis"][0]
        gr = {n: (d1[n][0] * ex, d1[n][1] * ir, d1[n][2] * irs) for n in "uvw"}
        om_h = om.clamp(min=1e-10)
        cn = (0.028 * k.clamp(min=0) ** 2 if p.turb_model == 1 else k.clamp(min=0)) / om_h
        cn = cn.clamp(max=1000.0 / (p.u_0 * p.L_atm))
        der = 0.66667 * (gr["u"][0] + gr["v"][1] + gr["w"][2])
        prod = torch.zeros_like(k)
        for q, n in enumerate("uvw"):
            prod = prod + (cn * (2 * gr[n][q] - der) - 0.66667 * k) * gr[n][q]
            for r, o in enumerate("uvw"):
                if r != q:
                    prod = prod + cn * (gr[n][r] + gr[o][q]) * gr[n][r]
        prod = prod.clamp(min=0)
        ks, oms = k.clamp(min=1e-10), om_h
        lim_o, lim_k = 20 * oms * oms, 20 * ks * oms
        cross = (d1["tke"][0] * d1["dis"][0] + d1["tke"][1] * d1["dis"][1] * ir ** 2
                 + d1["tke"][2] * d1["dis"][2] * irs ** 2)
        if p.turb_model == 1:
            dk, do = inv_re + nue, inv_re + nue / 1.3
            sk, so = prod - oms, 1.35 * oms / ks * prod - 1.8 * oms ** 2 / ks
        elif p.turb_model == 2:
            dk, do = inv_re + 0.6 * nue, inv_re + 0.5 * nue
            pk = torch.minimum(prod, 1.8 * ks * oms)
            sk = pk - 0.09 * ks * oms
            so = 0.52 * oms / ks * pk - 0.0708 * oms ** 2 + torch.where(cross <= 0, 0.0, 0.125) * cross / oms
        else:
            cd = (2 * 1.168 / om * cross).clamp(min=1e-20)
            arg = torch.minimum(torch.maximum(k.sqrt() / (0.09 * om * wall),
                                              500 * 1.5e-5 / (p.u_0 * p.L_atm) / (wall ** 2 * om)),
                                4 * 1.168 * k / (cd * wall ** 2))
            F = torch.tanh(arg ** 4)
            dk = inv_re + nue / (1.176 * F + 1 - F)
            do = inv_re + nue / (2 * F + 1.168 * (1 - F))
            pk = torch.minimum(prod, 1.8 * ks * oms)
            sk = pk - 0.09 * ks * oms
            so = ((0.413 * F + 0.2 * (1 - F)) * pk * oms / ks - (0.0333 * F + 0.0368 * (1 - F)) * oms ** 2
                  + 2 * (1 - F) * 1.168 / oms * cross)
        sk, so = torch.minimum(torch.maximum(sk, -lim_k), lim_k), torch.minimum(torch.maximum(so, -lim_o), lim_o)
        r = {"tke": -central("tke") + laplace("tke") * dk + sk, "dis": -central("dis") + laplace("dis") * do + so}
        nu = inv_re + nue
        metric = (1 + cs ** 2 / sn ** 2) * ir ** 2
        cot2 = 2 * cs / sn * ir * irs
        r["u"] = (-dp["r"] * ex - limited("u") + nu * (sum(second("u")) + 2 * U * ir ** 2 + 4 * d1["u"][0] * ir * ex
                                                      + d1["u"][1] * cs / sn * ir ** 2)
                  + 0.01 * p.g * DT / p.u_0 * (s["t"][0] - t_ref))
        r["v"] = (-dp["t"] * ir - limited("v") + nu * (laplace("v") - metric * V + 2 * d1["u"][1] * ir ** 2
                                                      - d1["w"][2] * cot2)
                  + force * 2 * cs * W + MCV * f["MC_v"][I] - drag * V)
        r["w"] = (-dp["p"] * irs - limited("w") + nu * (laplace("w") - metric * W + 2 * d1["u"][2] * ir * irs
                                                       + d1["v"][2] * cot2)
                  - force * 2 * cs * V + MCV * f["MC_w"][I] - drag * W)
        r["t"] = (p.u_0 ** 2 / (p.cp_l * p.t_0) * (ur * dp["r"] + vt * dp["t"] + wp * dp["p"]) - limited("t")
                  + laplace("t") * nu / p.pr_turb + source["t"] - k_T * (s["t"][0] - f["t_eq"][I]))
        for n in ("c", "cloud", "ice", "gr", "co2"):
            coef = inv_re / (p.sc_CO2 if n == "co2" else p.sc_WaterVapour)
            r[n] = -(limited(n) if n in ("c", "cloud", "ice") else central(n)) + laplace(n) * coef + source[n]
        return r, (prod, sk, so)

    y = {n: f[n] for n in Y}
    total = None
    for coef, weight in ((0.5 * DT, 1), (0.5 * DT, 2), (DT, 2), (DT / 6, 1)):
        r, turb = rhs(y)
        last = y
        total = r if total is None else {n: total[n] + weight * r[n] for n in Y}
        kk = total if weight == 1 and coef == DT / 6 else r
        y = {}
        for n in Y:
            v = f[n + "n"][I] + kk[n] * coef
            if n in ("c", "cloud", "ice", "gr"):
                v = v.clamp(min=0)
            elif n == "tke":
                v = v.clamp(0, 1000.0 / p.u_0 ** 2)
            elif n == "dis":
                v = v.clamp(min=1e-10)
            y[n] = f[n].clone()
            y[n][I] = v
    out = dict.fromkeys(_outputs("rk4", case))
    out.update(y)
    for n, c in zip(("u", "v", "w"), (dp["r"] * ex, dp["t"] * ir, dp["p"] * irs)):
        a = _fields(g, ("aux_" + n,))["aux_" + n]
        a[I] = r[n] + c
        out["aux_" + n] = a
    if case["diag"]:
        for n, x in zip(("prod", "tke_source", "dis_source"), turb):
            a = _fields(g, (n,))[n]
            a[I] = x
            out[n] = a
    else:
        out.update({n + "n": y[n] for n in Y})
    return out


def _exact_project(case, seed):
    g = _context(case, seed)
    p, m = g.params, _Grid(g)
    f = _fields(g, ("u", "v", "w"))
    I = (slice(1, -1),) * 3
    ex, ir, irs = m.exp[1:-1], m.ir[1:-1], m.irs[1:-1, 1:-1]
    u, v, w = (f[n].clone() for n in ("u", "v", "w"))
    for x in (u, v, w):            # the radial boundary copies the next level
        x[0, 1:-1, 1:-1], x[-1, 1:-1, 1:-1] = x[1, 1:-1, 1:-1], x[-2, 1:-1, 1:-1]
    n1, n2, n3 = ex ** 2 / m.dr ** 2, ir ** 2 / m.dthe ** 2, irs ** 2 / m.dphi ** 2
    den = 2 * (n1 + n2 + n3)
    su, sv, sw = _star(u), _star(v), _star(w)
    src = ((su[1] - su[2]) / (2 * m.dr) * ex + (sv[3] - sv[4]) / (2 * m.dthe) * ir + (sw[5] - sw[6]) / (2 * m.dphi) * irs)
    src = torch.minimum(torch.maximum(src, -2 * den), 2 * den)
    q = torch.zeros_like(u)
    red = sum(torch.meshgrid(*(torch.arange(1, n - 1, device="cuda") for n in g.shape), indexing="ij")) % 2 == 0
    for _ in range(case["sweeps"]):
        # the cells with even i + j + k first; a cell's neighbours are of the other colour
        for colour in (red, ~red):
            s = _star(q)
            q[I] = torch.where(colour, ((s[1] + s[2]) * n1 + (s[3] + s[4]) * n2 + (s[5] + s[6]) * n3 - src) / den, s[0])
        q[0, 1:-1, 1:-1], q[-1, 1:-1, 1:-1] = q[1, 1:-1, 1:-1], q[-2, 1:-1, 1:-1]
        q[:, 0, 1:-1], q[:, -1, 1:-1] = q[:, 1, 1:-1], q[:, -2, 1:-1]
        q[:, :, 0] = q[:, :, -1] = 0.5 * (q[:, :, 1] + q[:, :, -2])
        q.clamp_(-10.0, 10.0)
    s = _star(q)
    f["u"][I] -= (s[1] - s[2]) / (2 * m.dr) * ex
    f["v"][I] -= (s[3] - s[4]) / (2 * m.dthe) * ir
    f["w"][I] -= (s[5] - s[6]) / (2 * m.dphi) * irs
    return f


def _exact_radiation(case, seed):
    g = _context(case, seed)
    p, m = g.params, _Grid(g)
    f = _fields(g, ("t", "c", "co2", "cloud", "ice", "p_stat"))
    im, jm, _ = g.shape
    ps, t = f["p_stat"], f["t"]
    T = t * p.t_0
    dP = 100 * torch.cat([ps[:-1] - ps[1:], ps[-1:]]).clamp(min=0)
    dz = (m.height[1:].float() - m.height[:-1].float()).double()
    dz = torch.cat([dz, dz[-1:]])[:, None, None]
    qv, qc = f["c"].clamp(min=0), f["co2"].clamp(min=0)
    qb = (1 - qv - qc).clamp(min=0)
    tau = (p.kappa_H2O * qv + p.kappa_CO2 * qc + p.kappa_bg * qb) * dP / p.g * ps * 100 / 1e5
    R = qv * 8.314462618 / 0.018015 + qc * 8.314462618 / 0.044010 + qb * p.R_bg
    rho = ps * 100 / (R * T)
    lwp, iwp = f["cloud"].clamp(min=0) * rho * dz * 1e3, f["ice"].clamp(min=0) * rho * dz * 1e3
    tau = tau + 0.12 * lwp + 0.055 * iwp
    eps = torch.where(tau > 700, torch.ones_like(tau), -torch.expm1(-tau))
    cw = (lwp.sum(0) + 0.5 * iwp.sum(0)) / 100
    albedo = p.albedo_surface + max(0.0, p.albedo_cloud - p.albedo_surface) * cw / (cw + 2)
    jj = torch.arange(jm, dtype=torch.float64, device="cuda")
    half = (jm - 1) // 2
    x = torch.where(jj > half, jm - 1 - jj, jj) / half
    sw = ((p.rad_pole_short - p.rad_equator_short) * (x * x - 2 * x) + p.rad_pole_short)[:, None]
    Ts = T[0].clone()
    up, dn = torch.zeros_like(T), torch.zeros_like(T)
    for it in range(5):
        up[0] = p.sigma * Ts ** 4
        for i in range(1, im):
            up[i] = up[i - 1] * (1 - eps[i]) + eps[i] * p.sigma * T[i] ** 4
        d = torch.zeros_like(Ts)
        for i in range(im - 1, 0, -1):
            d = d * (1 - eps[i]) + eps[i] * p.sigma * T[i] ** 4
            dn[i] = d
        if it < 4:
            emit = 0.5 * (up[:-1] + torch.cat([dn[2:], torch.zeros_like(dn[:1])]))
            T[1:] = torch.where(emit > 0, (emit / p.sigma) ** 0.25, T[1:])
    k = 4 * p.sigma * Ts ** 3
    T[0] = ((1 - albedo) * sw + p.geothermal_flux + dn[1] - p.sigma * Ts ** 4 + k * Ts + 15.0 * T[1]) / (k + 15.0)
    up[0] = p.sigma * T[0] ** 4
    return {"t": t * 0.95 + T / p.t_0 * 0.05, "radiation": up, "epsilon": eps}
