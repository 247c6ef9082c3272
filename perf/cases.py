"""The framework's work as its users call it, at the sizes of its configurations, tests and benchmark.

Most cases are chemistry advances (``react`` on one box, ``react_boxes`` on all boxes of a level,
``advance_chemistry`` on PeleLM's MKS state); beside them stand the pointwise entries a PeleLM step
makes around the advance (T from rho h, instantaneous rates, the heat-release derive) and one
training step of the learned surrogate. ``draw`` spreads sizes, box shapes, mechanisms, precision
and options over the ranges the listed cases stand for.
"""
from __future__ import annotations

import json
import math
import os

import torch

from pelelm_gb300 import surrogate as sg
from pelelm_gb300.reactor import BoxArrays, ReactorBase, heat_release, reaction_rates, rhoh_to_temp

DEV = "cuda"
DATA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pelelm_gb300", "data")
R_ERG = 8.31446261815324e7   # erg/mol/K
R_CAL = R_ERG / 4.184e7      # cal/mol/K
P_ATM = 1.01325e6            # dyn/cm^2
RTOL, ATOL = 1e-6, 1e-10

# phi, T = T0 + c U[dT], p [atm] and fuel of the named configurations of pelelm_gb300/workloads.py
STATES = {
    "lidryer_syn": dict(fuel="H2", ox=1.88, o2=0.5, phi=(0.5, 2.0), dT=(900.0, 2100.0), p=(1.0, 1.0)),
    "drm19_syn": dict(fuel="CH4", ox=7.52, o2=2.0, phi=(0.6, 1.4), dT=(1900.0, 1900.0), p=(1.0, 1.0)),
    "gri_syn": dict(fuel="CH4", ox=7.52, o2=2.0, phi=(0.5, 1.5), dT=(2100.0, 2100.0), p=(1.0, 10.0)),
}
# operations of one right-hand side, and right-hand sides a cell takes over dt_react (rounded means
# of the configurations), for work()
RHS_FLOPS = {"lidryer_syn": 2068, "drm19_syn": 8252, "gri_syn": 28317}
RHS_PER_CELL = {"lidryer_syn": 50, "drm19_syn": 67, "gri_syn": 149}
# most cells of one drawn advance, by mechanism and precision: none costs more than the largest
# listed case
MAX_CELLS = {("lidryer_syn", "mixed"): 400000, ("lidryer_syn", "fp64"): 200000,
             ("drm19_syn", "mixed"): 200000, ("drm19_syn", "fp64"): 100000,
             ("gri_syn", "mixed"): 4096, ("gri_syn", "fp64"): 640}


def listed():
    return [
        # the smallest call: one 8^3 AMR box, waited for by the caller (react returns its failures)
        dict(name="react_lidryer_box8", op="react", mech="lidryer_syn", prec="mixed", boxes="8x8x8", dt=1e-5,
             forcing=True),
        # an ordinary single box of a plain-GPU run, no forcing, short dt_react
        dict(name="react_lidryer_box32", op="react", mech="lidryer_syn", prec="mixed", boxes="32x32x32", dt=1e-6,
             forcing=False),
        # all boxes of an AMR hierarchy in one advance, replayed from the reactor's CUDA graph
        dict(name="boxes_lidryer_amr", op="boxes", mech="lidryer_syn", prec="mixed",
             boxes="64x64x64,32x32x32*3,16x16x16*5,8x8x8*20", dt=1e-5, forcing=True, graph=True),
        # one ragged box of the 21-species mechanism, as the box loop of a 2-level run calls it
        dict(name="react_drm19_ragged", op="react", mech="drm19_syn", prec="mixed", boxes="13x9x7", dt=1e-5,
             forcing=True),
        # PeleLM's whole chemistry step: MKS state, covered cells masked, I_R, the GPU deck's tolerances
        dict(name="chem_drm19_deck", op="chem", mech="drm19_syn", prec="mixed",
             boxes="32x32x32,32x24x16*2,16x16x16*3,15x17x9*2", dt=1e-5, forcing=True, deck=True),
        # the benchmark's workload: surrogate with BDF fallback, 21 species, boxes of 16^3 and 32^3
        dict(name="boxes_drm19_surrogate", op="boxes", mech="drm19_syn", prec="mixed",
             boxes="32x32x32*4,16x16x16*16", dt=1e-5, forcing=True, graph=True, surrogate=True),
        # the reference's precision throughout
        dict(name="boxes_drm19_fp64", op="boxes", mech="drm19_syn", prec="fp64", boxes="32x32x16*2,16x16x16*4",
             dt=1e-5, forcing=True),
        # the 53-species mechanism, mixed precision with the FP64 retry of failed cells
        dict(name="boxes_gri_mixed", op="boxes", mech="gri_syn", prec="mixed", boxes="16x16x8,8x8x8*2", dt=1e-5,
             forcing=True),
        # instantaneous rates of a level's grid
        dict(name="rates_drm19", op="rates", mech="drm19_syn", boxes="128x64x48"),
        # T from (rho h, Y) after an advection step, the largest mechanism
        dict(name="rhoh_to_temp_gri", op="h2t", mech="gri_syn", boxes="96x64x33"),
        # the HeatRelease derive of a plot file
        dict(name="heat_release_lidryer", op="hr", mech="lidryer_syn", boxes="128x128x65"),
        # one optimiser step of the surrogate at its training batch
        dict(name="surrogate_train_step", op="train", batch=8192, n_in=44, n_out=20, width=256, depth=4),
    ]


# ---------------------------------------------------------------------- drawn cases
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_boxes(rng, cells):
    """Boxes of 4 to 32 cells a side (cubes of the AMR sizes, or ragged) with about `cells` cells."""
    out, left = [], cells
    while left >= 64 and len(out) < 60:
        top = max(4, min(32, int(round(left ** (1.0 / 3.0)))))
        if rng.random() < 0.4:
            s = max(v for v in (4, 8, 16, 32) if v <= top)
            d = (s, s, s)
        else:
            d = tuple(rng.randint(max(3, top // 2), top) for _ in range(3))
        n = max(1, min(left // (d[0] * d[1] * d[2]), rng.choice((1, 2, 4, 16))))
        out.append("%dx%dx%d" % d + ("*%d" % n if n > 1 else ""))
        left -= n * d[0] * d[1] * d[2]
    return ",".join(out)


def draw(rng):
    op = rng.choice(("react", "react", "boxes", "boxes", "boxes", "chem", "chem", "rates", "h2t", "hr", "train"))
    if op == "train":
        return dict(op=op, batch=32 * _log(rng, 8, 512), n_in=rng.randint(20, 44), n_out=rng.randint(9, 30),
                    width=rng.choice((64, 128, 256)), depth=rng.randint(2, 4))
    if op in ("rates", "h2t", "hr"):
        mech = rng.choice(("lidryer_syn", "drm19_syn") + (() if op == "rates" else ("gri_syn",)))
        n = _log(rng, 512, 500000 if mech == "drm19_syn" and op == "rates" else 1000000 // (4 if mech == "gri_syn" else 1))
        nx = rng.randint(5, 128)
        ny = max(1, min(128, int(round((n / nx) ** 0.5)) + rng.randint(-1, 1)))
        return dict(op=op, mech=mech, boxes="%dx%dx%d" % (nx, ny, max(1, n // (nx * ny))))
    mech = rng.choice(("lidryer_syn", "lidryer_syn", "drm19_syn", "drm19_syn", "gri_syn"))
    prec = rng.choice(("mixed", "mixed", "fp64"))
    most = MAX_CELLS[(mech, prec)]
    c = dict(op=op, mech=mech, prec=prec, dt=rng.choice((1e-6, 1e-5)), forcing=rng.random() < 0.75)
    if op == "react":
        n = _log(rng, 64, min(32768, most))
        nx = rng.randint(4, 32)
        ny = max(1, min(32, int(round((n / nx) ** 0.5))))
        c["boxes"] = "%dx%dx%d" % (nx, ny, max(1, min(n // (nx * ny), 32)))
        return c
    c["boxes"] = _draw_boxes(rng, _log(rng, 512, most))
    if op == "chem":
        c["deck"] = rng.random() < 0.3 and mech != "gri_syn"
    else:
        c["graph"] = rng.random() < 0.5
        c["surrogate"] = mech == "drm19_syn" and rng.random() < 0.3
    return c


# ---------------------------------------------------------------------- inputs
def _dims(case):
    out = []
    for part in case["boxes"].split(","):
        d, _, n = part.partition("*")
        out += [tuple(int(v) for v in d.split("x"))] * int(n or 1)
    return out


def _mech(name, device=DEV):
    with open(os.path.join(DATA, name + ".json")) as f:
        d = json.load(f)

    def t(v):
        return torch.tensor(v, dtype=torch.float64, device=device)

    return dict(json=d, names=[s["name"] for s in d["species"]], W=t([s["W"] for s in d["species"]]),
                Tmid=t([s["Tmid"] for s in d["species"]]), low=t([s["low"] for s in d["species"]]),
                high=t([s["high"] for s in d["species"]]))


def _thermo(m, T):
    """h/RT, cp/R and g/RT of every species at T: NASA-7, (n, ns)."""
    T = T[:, None]
    out = []
    for a in (m["low"], m["high"]):
        a = [a[None, :, i] for i in range(7)]
        h = a[0] + a[1] * T / 2 + a[2] * T ** 2 / 3 + a[3] * T ** 3 / 4 + a[4] * T ** 4 / 5 + a[5] / T
        cp = a[0] + a[1] * T + a[2] * T ** 2 + a[3] * T ** 3 + a[4] * T ** 4
        s = a[0] * torch.log(T) + a[1] * T + a[2] * T ** 2 / 2 + a[3] * T ** 3 / 3 + a[4] * T ** 4 / 4 + a[6]
        out.append((h, cp, h - s))
    cold = T < m["Tmid"][None]
    return [torch.where(cold, x, y) for x, y in zip(*out)]


def _h_mass(m, T):
    return _thermo(m, T)[0] * (R_ERG * T)[:, None] / m["W"][None]


def _states(m, mech, n, seed, dt, forcing):
    """The configurations' state distribution (phi, progress variable, radical seeds) and forcing,
    CGS, cell-major."""
    cfg = STATES[mech]
    g = torch.Generator(device=DEV).manual_seed(seed)

    def u(lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=torch.float64)

    ix = m["names"].index
    phi, c = u(*cfg["phi"]), u(0.0, 1.0)
    Xu = torch.zeros(n, len(m["names"]), device=DEV, dtype=torch.float64)
    Xb = Xu.clone()
    Xu[:, ix(cfg["fuel"])], Xu[:, ix("O2")], Xu[:, ix("N2")] = phi, cfg["o2"], cfg["ox"]
    burned = torch.clamp(phi, max=1.0)
    Xb[:, ix(cfg["fuel"])] = phi - burned
    Xb[:, ix("O2")] = cfg["o2"] * (1.0 - burned)
    Xb[:, ix("N2")] = cfg["ox"]
    if cfg["fuel"] == "CH4":
        Xb[:, ix("CO2")], Xb[:, ix("H2O")] = burned, 2.0 * burned
    else:
        Xb[:, ix("H2O")] = burned
    Yu, Yb = Xu * m["W"], Xb * m["W"]
    Y = (1.0 - c)[:, None] * Yu / Yu.sum(1, True) + c[:, None] * Yb / Yb.sum(1, True)
    for r in ("H", "O", "OH"):
        Y[:, ix(r)] += 1e-6
    Y /= Y.sum(1, True)
    T = 300.0 + c * u(*cfg["dT"])
    rho = P_ATM * u(*cfg["p"]) / (R_ERG * T * (Y / m["W"]).sum(1))
    rY = rho[:, None] * Y
    rE = rho * (Y * _h_mass(m, T)).sum(1)
    F, Fh = torch.zeros_like(rY), torch.zeros_like(T)
    if forcing:
        F = torch.randn(n, rY.shape[1], generator=g, device=DEV, dtype=torch.float64) * 0.1
        F = torch.maximum(F, -0.5 * rY / dt)       # drains at most half of a species over dt_react
        F -= F.sum(1, True) * Y                    # no net mass
        Fh = torch.randn(n, generator=g, device=DEV, dtype=torch.float64) * 1e9
    return rY, T, rE, F, Fh, u(0.0, 1.0)


def _arena(dims, a):
    """(ncell, ncomp) -> one buffer holding a component-major block for each box, and its views."""
    a = a if a.dim() == 2 else a[:, None]
    flat = torch.empty(a.numel(), dtype=a.dtype, device=a.device)
    views, c, o = [], 0, 0
    for nx, ny, nz in dims:
        n = nx * ny * nz
        v = flat[o:o + n * a.shape[1]].view(a.shape[1], nz, ny, nx)
        v.copy_(a[c:c + n].T.reshape(v.shape))
        views.append(v)
        c, o = c + n, o + n * a.shape[1]
    return flat, views


def prepare(case, seed):
    op = case["op"]
    if op == "train":
        m = sg.SurrogateMLP(torch, case["n_in"], case["n_out"], width=case["width"], depth=case["depth"], seed=seed)
        g = torch.Generator(device=DEV).manual_seed(seed)
        x = torch.randn(case["batch"], case["n_in"], generator=g, device=DEV)
        T = torch.zeros(case["batch"], m.n_out_pad, device=DEV)
        T[:, :case["n_out"]] = torch.randn(case["batch"], case["n_out"], generator=g, device=DEV)
        return dict(case=case, mlp=m, X=m.prepare_input(x), T=T)
    dims, mech = _dims(case), case["mech"]
    m = _mech(mech)
    ncell = sum(a * b * c for a, b, c in dims)
    dt = case.get("dt", 1e-5)
    rY, T, rE, F, Fh, cover = _states(m, mech, ncell, seed, dt, case.get("forcing", False))
    s = dict(case=case, dims=dims, mech=mech, dt=dt)
    if op in ("rates", "h2t", "hr"):
        rho = rY.sum(1)
        if op == "hr":  # rates of a reacting field: production and destruction of every species
            g = torch.Generator(device=DEV).manual_seed(seed + 1)
            rY = torch.randn(rY.shape, generator=g, device=DEV, dtype=torch.float64) * 1e2
        else:
            rY = rY * 1e3
        s["box"] = ((0, 0, 0), tuple(d - 1 for d in dims[0]))
        for k, v in (("rY", rY), ("T", T), ("rE", rE * 0.1)):
            s[k + "_flat"], (s[k],) = _arena(dims, v)
        if op == "h2t":  # the old temperature is the guess, the energy has moved on
            s["rE_flat"] += 0.1 * (rho * 1e3) * 4e4 * (cover - 0.5)
            s["guess"] = s["T_flat"].clone()
        s["out_flat"], (s["out"],) = _arena(dims, torch.zeros_like(rY if op == "rates" else T))
        return s
    if op == "chem":
        rY, F, rE, Fh = rY * 1e3, F * 1e3, rE * 0.1, Fh * 0.1
    n_old = rY.numel() + 2 * ncell
    new = torch.empty(n_old, device=DEV, dtype=torch.float64)  # rhoY | T | rho h, one copy restores all
    views, o = {}, 0
    old = []
    for k, v in (("rY", rY), ("T", T), ("rE", rE)):
        flat, _ = _arena(dims, v)
        old.append(flat)
        seg = new[o:o + flat.numel()]
        s[k + "_flat"], o = seg, o + flat.numel()
        nc, c, vs = (v.shape[1] if v.dim() == 2 else 1), 0, []
        for nx, ny, nz in dims:
            n = nx * ny * nz * nc
            vs.append(seg[c:c + n].view(nc, nz, ny, nx))
            c += n
        views[k] = vs
    s["old"], s["new"] = torch.cat(old), new
    s["F_flat"], views["F"] = _arena(dims, F)
    s["Fh_flat"], views["Fh"] = _arena(dims, Fh)
    s["FC_flat"], views["FC"] = _arena(dims, torch.zeros(ncell, device=DEV, dtype=torch.float64))
    views["mask"] = [None] * len(dims)
    if op == "chem":  # a tenth of the cells are covered by a finer level
        s["mask_flat"], views["mask"] = _arena(dims, torch.where(cover < 0.1, -1, 1).to(torch.int32))
        s["IR_flat"], s["IR"] = _arena(dims, torch.zeros_like(F))
    s["boxes"] = [BoxArrays(((0, 0, 0), (d[0] - 1, d[1] - 1, d[2] - 1)), views["rY"][b], views["F"][b], views["T"][b],
                            views["rE"][b], views["Fh"][b], views["FC"][b], views["mask"][b]) for b, d in enumerate(dims)]
    opts = [f"gb.precision={case['prec']}", f"ode.rtol={RTOL}"]
    if case.get("deck"):  # the GPU decks' settings: tolerances on typical values, order 4, GMRES key
        opts += ["ode.atol=1e-5", "peleLM.use_typ_vals_chem=1", "cvode.max_order=4", "cvode.solve_type=GMRES"]
    else:
        opts += [f"ode.atol={ATOL}"]
    if mech == "gri_syn":
        opts += ["ode.max_steps=2000"]
    if case.get("graph"):
        opts += ["gb.graph=1"]
        s["stream"] = torch.cuda.Stream()
    if case.get("surrogate"):
        opts += [f"gb.surrogate={os.path.join(DATA, mech + '.pgbs')}"]
    s["reactor"] = ReactorBase.create("ReactorCvode", mech, " ".join(opts))
    s["reactor"].init(2, 1)
    if case.get("deck"):
        k = 1e-3 if op == "chem" else 1.0
        typ = [max(1e-10, k * float(v)) for v in (rY.amax(0) - rY.amin(0)).tolist()]
        s["reactor"].set_typ_vals_ode(typ + [float(T.max() - T.min())])
    return s


# ---------------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "train":
        loss = s["mlp"].train_step(s["X"], s["T"])
        return dict(loss=loss, W=s["mlp"].W, b=s["mlp"].b)
    if op == "rates":
        reaction_rates(s["mech"], s["box"], s["rY"], s["rE"], s["T"], None, s["out"])
        return dict(rhoYdot=s["out_flat"])
    if op == "hr":
        heat_release(s["mech"], s["box"], s["T"], s["rY"], s["out"])
        return dict(hr=s["out_flat"])
    if op == "h2t":
        s["T_flat"].copy_(s["guess"])
        rhoh_to_temp(s["mech"], s["box"], s["rY"], s["rE"], s["T"])
        return dict(T=s["T_flat"])
    out = dict(rY=s["rY_flat"], T=s["T_flat"], rE=s["rE_flat"], FC=s["FC_flat"])
    if op == "react":
        s["new"].copy_(s["old"])
        b = s["boxes"][0]
        out["nfail"] = s["reactor"].react(b.box, b.rY, b.rY_src, b.T, b.rEner, b.rEner_src, b.FC, b.mask, s["dt"], 0.0)
    elif op == "chem":
        s["new"].copy_(s["old"])
        s["reactor"].advance_chemistry(s["boxes"], s["dt"], I_R=s["IR"])
        out["I_R"] = s["IR_flat"]
    elif "stream" in s:
        s["stream"].wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s["stream"]):
            s["new"].copy_(s["old"])
            s["reactor"].react_boxes(s["boxes"], s["dt"], stream=s["stream"])
        torch.cuda.current_stream().wait_stream(s["stream"])
    else:
        s["new"].copy_(s["old"])
        s["reactor"].react_boxes(s["boxes"], s["dt"])
    return out


def work(case):
    op = case["op"]
    if op == "train":
        dims = [2 * ((case["n_in"] + 15) // 16 * 16)] + [case["width"]] * case["depth"] + [(case["n_out"] + 31) // 32 * 32]
        nw = sum(a * b for a, b in zip(dims, dims[1:]))
        return dict(bytes=case["batch"] * (2 * dims[0] + 4 * dims[-1]) + 32 * nw, flops=6 * case["batch"] * nw)
    n = sum(a * b * c for a, b, c in _dims(case))
    ns = {"lidryer_syn": 9, "drm19_syn": 21, "gri_syn": 53}[case["mech"]]
    if op == "rates":
        return dict(bytes=8 * n * (2 * ns + 2), flops=n * RHS_FLOPS[case["mech"]])
    if op == "h2t":
        return dict(bytes=8 * n * (ns + 3), flops=n * 3 * 22 * ns)
    if op == "hr":
        return dict(bytes=8 * n * (ns + 2), flops=n * 13 * ns)
    io = 3 * ns + 6 + (ns if op == "chem" else 0)
    evals = RHS_PER_CELL[case["mech"]] * (1.0 if case["dt"] > 5e-6 else 0.5)
    return dict(bytes=8 * n * (io + 2 * (ns + 2)), flops=n * evals * RHS_FLOPS[case["mech"]])


# ---------------------------------------------------------------------- the same in 64 bits
def _newton_T(m, h, Y, T):
    for _ in range(60):
        hRT, cpR, _ = _thermo(m, T)
        f = h - (Y * hRT * (R_ERG * T)[:, None] / m["W"]).sum(1)
        T = T + torch.clamp(f / (Y * cpR * R_ERG / m["W"]).sum(1), -100.0, 100.0)
    return T


def _production(m, T, C):
    """Molar production rates [mol/cm^3/s]: modified Arrhenius, third bodies, Lindemann/Troe
    fall-off, reverse rates from K_c."""
    ix = m["names"].index
    g = _thermo(m, T)[2]
    wdot = torch.zeros_like(C)
    ctot = C.sum(1)
    for r in m["json"]["reactions"]:
        def k(a):
            return a["A"] * T ** a["beta"] * torch.exp(-a["Ea"] / (R_CAL * T))
        kf = k(r["rate"])
        M = ctot + sum((e - 1.0) * C[:, ix(s)] for s, e in r["efficiencies"].items()) if r["kind"] != "elementary" else 1.0
        if r["kind"] == "falloff":
            Pr = k(r["low"]) * M / kf
            F = 1.0
            if r["troe"]:
                a, T3, T1 = r["troe"][:3]
                Fc = (1.0 - a) * torch.exp(-T / T3) + a * torch.exp(-T / T1)
                if len(r["troe"]) > 3:
                    Fc = Fc + torch.exp(-r["troe"][3] / T)
                lF = torch.log10(Fc)
                lP = torch.log10(torch.clamp(Pr, min=1e-300)) - 0.4 - 0.67 * lF
                F = 10.0 ** (lF / (1.0 + (lP / (0.75 - 1.27 * lF - 0.14 * lP)) ** 2))
            kf = kf * Pr / (1.0 + Pr) * F
        q = kf.clone()
        for s, nu in r["reactants"].items():
            q = q * C[:, ix(s)] ** nu
        if r["reversible"]:
            dg = sum(nu * g[:, ix(s)] for s, nu in r["products"].items()) - sum(nu * g[:, ix(s)] for s, nu in r["reactants"].items())
            dnu = sum(r["products"].values()) - sum(r["reactants"].values())
            back = kf * torch.exp(torch.clamp(dg - dnu * torch.log(P_ATM / (R_ERG * T)), max=700.0))
            for s, nu in r["products"].items():
                back = back * C[:, ix(s)] ** nu
            q = q - back
        if r["kind"] == "three_body":
            q = q * M
        for s, nu in r["reactants"].items():
            wdot[:, ix(s)] -= nu * q
        for s, nu in r["products"].items():
            wdot[:, ix(s)] += nu * q
    return wdot


def exact(case, seed):
    op = case["op"]
    if op in ("react", "boxes", "chem"):
        return None  # an integration to round-off takes far longer than 20 s
    s = prepare(case, seed)
    if op == "train":
        return _exact_train(case, s)
    m = _mech(case["mech"])
    nc = len(m["names"])
    n = s["T_flat"].numel()
    rY, T, rE = s["rY_flat"].view(nc, n).T, s["T_flat"], s["rE_flat"]
    if op == "hr":
        out = torch.cat([-(rY[i:i + 65536] * _h_mass(m, T[i:i + 65536]) * 1e-4).sum(1) for i in range(0, n, 65536)])
        return dict(hr=out)
    rho = rY.sum(1)
    out = []
    for i in range(0, n, 65536):
        Y = (rY[i:i + 65536] / rho[i:i + 65536, None])
        Tn = _newton_T(m, rE[i:i + 65536] / rho[i:i + 65536] * 1e4, Y, T[i:i + 65536])
        if op == "rates":
            out.append(_production(m, Tn, rho[i:i + 65536, None] * 1e-3 * Y / m["W"]) * m["W"] * 1e3)
        else:
            out.append(Tn)
    out = torch.cat(out)
    return dict(T=out) if op == "h2t" else dict(rhoYdot=out.T.reshape(-1))


def _exact_train(case, s):
    """Forward, backward and the first Adam step on the network's BF16 weights and inputs, with
    nothing else rounded."""
    m, lr, eps = s["mlp"], 1e-3, 1e-8
    W = [w.to(torch.bfloat16).double().requires_grad_() for w in m.W]
    b = [v.double().requires_grad_() for v in m.b]
    X = s["X"].double()
    x = X[:, :m.k_half] + X[:, m.k_half:2 * m.k_half]
    for i in range(len(W)):
        x = x @ W[i].T + b[i]
        if i + 1 < len(W):
            x = torch.nn.functional.gelu(x, approximate="tanh")
    d = (x - s["T"].double())[:, :case["n_out"]]
    (d.square().sum() / (case["batch"] * case["n_out"])).backward()
    step = [[(v.double() - lr * p.grad / (p.grad.abs() + eps)) for v, p in zip(vs, ps)] for vs, ps in ((m.W, W), (m.b, b))]
    return dict(loss=d.square().sum().reshape(1).detach(), W=step[0], b=step[1])
