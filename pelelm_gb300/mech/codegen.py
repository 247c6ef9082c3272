"""CUDA code generator for a mechanism: one header per mechanism with fully unrolled
production rates, reactor right-hand side and analytic Jacobian.

Plays the role FUEGO plays for PelePhysics (``Docs/source/manual/Model.rst:296-310``:
mechanism-specific generated rate/thermo code), written from scratch for sm_103a:

* all mechanism constants are folded into immediates (ln A, Ea/R, 1/W, NASA-7 with the
  per-species coefficient set picked by a predicated select, never a divergent branch);
* rates evaluate ln k in FP64 FMAs and take one exponential per coefficient;
* the Jacobian is a template on its arithmetic type: ``float`` recomputes every rate
  coefficient in FP32 (the inexact-Newton preconditioner), ``double`` gives the plain
  FP64 Jacobian. It writes J(i,k) at strides the caller gives, so the caller decides where the
  matrix lives (shared memory per thread or per cell).

The formulas are those of the CPU oracle (``oracle/chem_oracle.cpp``), which is the
equation-level restatement of Model.rst:227-296.
"""
from __future__ import annotations

import math
import os
import struct
from fractions import Fraction
from typing import Dict, List

from .model import Mechanism, R_CAL, R_ERG, P_ATM

LN10 = math.log(10.0)


def _f(x: float) -> str:
    r = repr(float(x))
    if "e" not in r and "." not in r and "inf" not in r and "nan" not in r:
        r += ".0"
    return r


class _Emitter:
    def __init__(self):
        self.lines: List[str] = []
        self.ind = 0

    def __call__(self, s: str = ""):
        self.lines.append("  " * self.ind + s if s else "")

    def text(self) -> str:
        return "\n".join(self.lines) + "\n"


def _thermo_select(e: _Emitter, m: Mechanism, prec: str):
    """Emit per-species NASA-7 coefficient selects a{k}_{i} for the current T."""
    tmids = sorted({s.Tmid for s in m.species})
    for t in tmids:
        e(f"const bool lo_{int(t)} = T < {_f(t)};")
    cast = "" if prec == "double" else "f"
    for k, s in enumerate(m.species):
        for i in range(7):
            lo, hi = s.low[i], s.high[i]
            e(f"const {prec} a{k}_{i} = lo_{int(s.Tmid)} ? {_f(lo)}{cast} : {_f(hi)}{cast};")


def _sel(lo_flag: str, lo: float, hi: float, prec: str = "double") -> str:
    """Predicated select between two folded immediates (no branch)."""
    if prec == "double":
        return f"({lo_flag} ? {_f(lo)} : {_f(hi)})"
    return f"({lo_flag} ? R({_f(lo)}) : R({_f(hi)}))"


def _g_expr(k, s, lo_flag):
    """g/RT = a0 (1-lnT) - a1 T/2 - a2 T^2/6 - a3 T^3/12 - a4 T^4/20 + a5/T - a6 (FP64, 6 FMA)."""
    L, H = s.low, s.high
    c = lambda i, f: _sel(lo_flag, L[i] * f, H[i] * f)
    return (f"fma({c(0, 1.0)}, lnT1, fma(T, fma(T, fma(T, fma(T, {c(4, -0.05)}, {c(3, -1.0 / 12.0)}), "
            f"{c(2, -1.0 / 6.0)}), {c(1, -0.5)}), fma({c(5, 1.0)}, invT, {c(6, -1.0)})))")


def _hW_expr(s, lo_flag, scale):
    """scale * h/RT (FP64, 5 FMA)."""
    L, H = s.low, s.high
    c = lambda i, f: _sel(lo_flag, L[i] * f * scale, H[i] * f * scale)
    return (f"fma(T, fma(T, fma(T, fma(T, {c(4, 0.2)}, {c(3, 0.25)}), {c(2, 1.0 / 3.0)}), {c(1, 0.5)}), "
            f"fma({c(5, 1.0)}, invT, {c(0, 1.0)}))")


def _cpW_expr(s, lo_flag, scale):
    """scale * cp/R (FP64, 4 FMA)."""
    L, H = s.low, s.high
    c = lambda i: _sel(lo_flag, L[i] * scale, H[i] * scale)
    return f"fma(T, fma(T, fma(T, fma(T, {c(4)}, {c(3)}), {c(2)}), {c(1)}), {c(0)})"


def check_supported(m: Mechanism) -> None:
    """The kernels take every reverse rate from K_c; explicit reverse Arrhenius parameters
    (CHEMKIN REV, which the reader keeps) are refused here rather than silently ignored."""
    for j, r in enumerate(m.reactions):
        if r.rev is not None:
            raise ValueError(f"{m.name}: reaction {j} ({r.equation()}) has explicit reverse parameters "
                             "(REV), which the rate kernels do not evaluate")


def total_only(m: Mechanism) -> set:
    """Species whose concentration enters the sum [M] alone; the exact form fuses its product there."""
    return {k for k, s in enumerate(m.species)
            if not any(s.name in r.reactants or s.name in r.products or r.efficiencies.get(s.name, 1.0) != 1.0
                       for r in m.reactions)}


def fused_third_body(m: Mechanism) -> int:
    """The reaction whose product q [M] the exact form fuses into the production rates: the last one, if
    it is a third-body reaction (-1: none). With total_only the contractions that the built-in mechanism's
    code had before its roundings were written out."""
    return m.nr - 1 if m.nr and m.reactions[-1].kind == "three_body" else -1


def gen_header(m: Mechanism) -> str:
    check_supported(m)
    ns, nr = m.ns, m.nr
    N = ns + 1
    W = [s.W for s in m.species]
    idx = {s.name: i for i, s in enumerate(m.species)}
    lnP0_R = math.log(P_ATM / R_ERG)  # ln(P0/R); ln(P0/RT) = lnP0_R - lnT
    e = _Emitter()
    guard = f"PGB_MECH_{m.name.upper()}_CUH"
    e("// GENERATED by pelelm_gb300/mech/codegen.py from pelelm_gb300/data/" + m.name + ".json.")
    e("// Do not edit. " + ("SYNTHETIC structure-matched mechanism." if m.synthetic else ""))
    e(f"#ifndef {guard}")
    e(f"#define {guard}")
    e('#include "../mech_common.cuh"')
    const_tab = constant_tables(m)
    if const_tab:
        e(f'#include "tab_{m.name}.cuh"')
    e(f'#include "tabg_{m.name}.cuh"')
    e()
    e("namespace pgb {")
    e(f"struct Mech_{m.name} {{")
    e.ind += 1
    e(f"using Tab = {'tab' if const_tab else 'tabg'}_{m.name}::Tables;  // per-thread kernels")
    e(f"using TabG = tabg_{m.name}::Tables;  // warp-per-cell kernel")
    e(f"static constexpr int NS = {ns};")
    e(f"static constexpr int NR = {nr};")
    e(f"static constexpr int N = {N};")
    e(f'static constexpr const char* NAME = "{m.name}";')
    e(f"static constexpr bool SYNTHETIC = {'true' if m.synthetic else 'false'};")
    e("// small mechanisms use the unrolled RHS / Jacobian below, larger ones the table-driven loops")
    e(f"static constexpr bool JAC_TABLE = {'true' if ns > 12 else 'false'};")
    e(f"static constexpr bool RHS_TABLE = {'true' if ns > 12 else 'false'};")
    e()
    # ---------------------------------------------------------------- molecular weights
    e("__host__ __device__ static constexpr double W(int k) {")
    e("  return " + " ".join(f"k == {k} ? {_f(w)} :" for k, w in enumerate(W)) + " 0.0;")
    e("}")
    e()
    # ---------------------------------------------------------------- thermo (mixture h, cp)
    e("// Mixture mass enthalpy [erg/g] and cp [erg/g/K] at T for mass fractions Y.")
    e("__device__ __forceinline__ static void h_cp_mix(const double T, const double* __restrict__ Y, double& h, double& cp) {")
    e.ind += 1
    e("const double invT = 1.0 / T;")
    for t in sorted({s.Tmid for s in m.species}):
        e(f"const bool lo_{int(t)} = T < {_f(t)};")
    e("double hs = 0.0, cps = 0.0;")
    for k, sp in enumerate(m.species):
        lf = f"lo_{int(sp.Tmid)}"
        e(f"hs = fma(Y[{k}], {_hW_expr(sp, lf, 1.0 / W[k])}, hs);")
        e(f"cps = fma(Y[{k}], {_cpW_expr(sp, lf, 1.0 / W[k])}, cps);")
    e(f"h = hs * ({_f(R_ERG)} * T);")
    e(f"cp = cps * {_f(R_ERG)};")
    e.ind -= 1
    e("}")
    e()
    # ---------------------------------------------------------------- FP64 rates core
    def plus_EaRT(ear, lnA):
        return f"fma({_f(-ear)}, invT, {_f(lnA)})" if ear != 0 else _f(lnA)

    def emit_rates_fp64(with_energy: bool):
        """Emit body computing q{j} from T, lnT, invT, C{k}, g{k} (FP64)."""
        # third-body concentrations
        needM = any(r.kind != "elementary" for r in m.reactions)
        if needM:
            e("const double Ctot = " + " + ".join(f"C{k}" for k in range(ns)) + ";")
        e(f"const double lnP0RT = {_f(lnP0_R)} - lnT;")
        for j, r in enumerate(m.reactions):
            e(f"// R{j}: {r.equation()}")
            lnA = math.log(r.rate.A)
            ear = r.rate.Ea / R_CAL
            e(f"double q{j};")
            e("{")
            e.ind += 1
            # A as a factor: added to the exponent (near 30) it would cost the rate ten roundings
            if r.kind == "falloff":
                e(f"const double lnkf = fma({_f(r.rate.beta)}, lnT, {plus_EaRT(ear, lnA)});")
            else:
                beta, ear_T = _f(r.rate.beta), f"{_f(-ear)} * invT"
                e("const double lnkfA = " + (f"{beta} * lnT;" if ear == 0 else f"fma({beta}, lnT, {ear_T});"))
            if r.kind != "elementary":
                terms = "Ctot"
                for sname, eff in r.efficiencies.items():
                    if eff != 1.0:
                        terms = f"fma({_f(eff - 1.0)}, C{idx[sname]}, {terms})"
                e(f"const double M = {terms};")
            if r.kind == "falloff":
                lnA0 = math.log(r.low.A)
                ear0 = r.low.Ea / R_CAL
                e(f"const double lnk0 = fma({_f(r.low.beta)}, lnT, {plus_EaRT(ear0, lnA0)});")
                # Pr = k0 M / kinf
                e("const double Pr = M * pgb_exp(lnk0 - lnkf);")
                if r.troe:
                    a, T3, T1 = r.troe[:3]
                    fc = f"fma({_f(1.0 - a)}, pgb_exp(T * {_f(-1.0 / T3)}), {_f(a)} * pgb_exp(T * {_f(-1.0 / T1)}))"
                    if len(r.troe) > 3:
                        fc = f"{fc} + pgb_exp(invT * {_f(-r.troe[3])})"
                    e(f"const double Fcent = {fc};")
                    e(f"const double lFc = pgb_log(Fcent) * {_f(1.0 / LN10)};")
                    e("const double cc = fma(-0.67, lFc, -0.4), nn = fma(-1.27, lFc, 0.75);")
                    e(f"const double lPr = pgb_log(fmax(Pr, 1e-300)) * {_f(1.0 / LN10)} + cc;")
                    e("const double f1 = lPr / fma(-0.14, lPr, nn);")
                    e(f"const double Fb = pgb_exp({_f(LN10)} * lFc / fma(f1, f1, 1.0));")
                    e("const double blend = Pr / (1.0 + Pr) * Fb;")
                else:
                    e("const double blend = Pr / (1.0 + Pr);")
                e("const double kf = pgb_exp(lnkf) * blend;")
            else:
                e(f"const double kf = {_f(r.rate.A)} * pgb_exp(lnkfA);")
            pf = " * ".join(f"C{idx[s]}" for s, nu in r.reactants.items() for _ in range(nu))
            pr = " * ".join(f"C{idx[s]}" for s, nu in r.products.items() for _ in range(nu))
            if r.reversible:
                dg = []
                for s, nu in r.products.items():
                    dg.append(("+" if nu == 1 else f"+ {nu}.0 *") + f" g{idx[s]}")
                for s, nu in r.reactants.items():
                    dg.append(("-" if nu == 1 else f"- {nu}.0 *") + f" g{idx[s]}")
                dnu = sum(r.products.values()) - sum(r.reactants.values())
                dgs = " ".join(dg).lstrip("+ ").strip()
                if dnu != 0:
                    dgs += f" - {_f(dnu)} * lnP0RT"
                # exponent capped at 700: exp stays finite, so an absent product (Pp = 0)
                # gives a zero reverse term instead of inf * 0 = NaN
                e(f"const double kr = kf * pgb_exp(fmin({dgs}, 700.0));")
                e(f"q{j} = fma(kf, {pf}, -kr * {pr});")
            else:
                e(f"q{j} = kf * {pf};")
            if r.kind == "three_body":
                e(f"q{j} *= M;")
            e.ind -= 1
            e("}")
        # production rates
        for k in range(ns):
            terms = []
            for j, r in enumerate(m.reactions):
                nu = r.products.get(m.species[k].name, 0) - r.reactants.get(m.species[k].name, 0)
                if nu != 0:
                    terms.append((nu, j))
            if not terms:
                e(f"const double wd{k} = 0.0;")
                continue
            expr = ""
            for nu, j in terms:
                if expr == "":
                    expr = (f"q{j}" if nu == 1 else (f"-q{j}" if nu == -1 else f"{_f(nu)} * q{j}"))
                else:
                    expr = (f"{expr} + q{j}" if nu == 1 else
                            (f"{expr} - q{j}" if nu == -1 else f"fma({_f(nu)}, q{j}, {expr})"))
            e(f"const double wd{k} = {expr};")

    def emit_rates_exact():
        """The same from y, C{k} and g{k} with every rounding written out: the lane-parallel evaluation
        (rate_of_progress_unrolled and group_rhs, csrc/bdf_group_kernel.cuh) performs these operations in
        this order, so the two agree bit for bit whatever the compiler would contract."""
        alone = total_only(m)
        if any(r.kind != "elementary" for r in m.reactions):
            tot = "C0"
            for k in range(1, ns):
                tot = f"fma(y[{k}], {_f(1.0 / W[k])}, {tot})" if k in alone else f"__dadd_rn({tot}, C{k})"
            e(f"const double Ctot = {tot};")
        e(f"const double lnP0RT = {_f(lnP0_R)} - lnT;")

        def product(first, names):
            for n_ in names:
                first = f"__dmul_rn({first}, {n_})" if first else n_
            return first

        for j, r in enumerate(m.reactions):
            e(f"// R{j}: {r.equation()}")
            e(f"double q{j};")
            if j == fused_third_body(m):
                e(f"double qu{j}, M{j};  // q{j} = qu{j} M{j}")
            e("{")
            e.ind += 1
            e(f"const double lnkf = fma({_f(r.rate.beta)}, lnT, fma({_f(-r.rate.Ea / R_CAL)}, invT, {_f(math.log(r.rate.A))}));")
            if r.kind != "elementary":
                terms = "Ctot"
                for sname, eff in r.efficiencies.items():
                    if eff != 1.0:
                        terms = f"fma({_f(eff - 1.0)}, C{idx[sname]}, {terms})"
                e(f"const double M = {terms};")
            if r.kind == "falloff":
                e(f"const double lnk0 = fma({_f(r.low.beta)}, lnT, fma({_f(-r.low.Ea / R_CAL)}, invT, {_f(math.log(r.low.A))}));")
                e("const double Pr = __dmul_rn(M, pgb_exp(lnk0 - lnkf));")
                e("double blend = Pr / __dadd_rn(1.0, Pr);")
                if r.troe:
                    a, T3, T1 = r.troe[:3]
                    fc = f"fma({_f(1.0 - a)}, pgb_exp(T * {_f(-1.0 / T3)}), __dmul_rn({_f(a)}, pgb_exp(T * {_f(-1.0 / T1)})))"
                    if len(r.troe) > 3:
                        fc = f"__dadd_rn({fc}, pgb_exp(invT * {_f(-r.troe[3])}))"
                    e(f"const double lFc = __dmul_rn(pgb_log({fc}), {_f(1.0 / LN10)});")
                    e("const double cc = fma(-0.67, lFc, -0.4), nn = fma(-1.27, lFc, 0.75);")
                    e(f"const double lPr = fma(pgb_log(fmax(Pr, 1e-300)), {_f(1.0 / LN10)}, cc);")
                    e("const double f1 = lPr / fma(-0.14, lPr, nn);")
                    e(f"blend = __dmul_rn(blend, pgb_exp(__dmul_rn({_f(LN10)}, lFc) / fma(f1, f1, 1.0)));")
                e("const double kf = __dmul_rn(pgb_exp(lnkf), blend);")
            else:
                e("const double kf = pgb_exp(lnkf);")
            pf = product("", [f"C{idx[s]}" for s, nu in r.reactants.items() for _ in range(nu)])
            if r.reversible:
                dg = ""
                for side, sign in ((r.products, 1), (r.reactants, -1)):
                    for s, nu in side.items():
                        g = f"g{idx[s]}"
                        if not dg:
                            dg = g if nu == 1 else f"__dmul_rn({nu}.0, {g})"
                        elif nu == 1:
                            dg = f"__d{'add' if sign > 0 else 'sub'}_rn({dg}, {g})"
                        else:
                            dg = f"fma({sign * nu}.0, {g}, {dg})"
                dnu = sum(r.products.values()) - sum(r.reactants.values())
                if dnu != 0:
                    dg = f"fma({_f(-dnu)}, lnP0RT, {dg})"
                # exponent capped at 700: exp stays finite, so an absent product (Pp = 0)
                # gives a zero reverse term instead of inf * 0 = NaN
                e(f"const double kr = -__dmul_rn(kf, pgb_exp(fmin({dg}, 700.0)));")
                pr = product("kr", [f"C{idx[s]}" for s, nu in r.products.items() for _ in range(nu)])
                e(f"q{j} = fma(kf, {pf}, {pr});")
            else:
                e(f"q{j} = __dmul_rn(kf, {pf});")
            if j == fused_third_body(m):
                e(f"qu{j} = q{j};")
                e(f"M{j} = M;")
            if r.kind == "three_body":
                e(f"q{j} = __dmul_rn(q{j}, M);")
            e.ind -= 1
            e("}")
        for k in range(ns):
            expr = ""
            for j, r in enumerate(m.reactions):
                nu = r.products.get(m.species[k].name, 0) - r.reactants.get(m.species[k].name, 0)
                if nu == 0:
                    continue
                if expr and abs(nu) == 1 and j == fused_third_body(m):
                    expr = f"fma({'-' if nu < 0 else ''}qu{j}, M{j}, {expr})"
                elif abs(nu) == 1:
                    expr = f"__d{'add' if nu > 0 else 'sub'}_rn({expr}, q{j})" if expr else ("q" if nu > 0 else "-q") + str(j)
                else:
                    expr = f"fma({_f(nu)}, q{j}, {expr})" if expr else f"__dmul_rn({_f(nu)}, q{j})"
            e(f"const double wd{k} = {expr or '0.0'};")

    def emit_gibbs():
        for t in sorted({s.Tmid for s in m.species}):
            e(f"const bool lo_{int(t)} = T < {_f(t)};")
        e("const double lnT1 = 1.0 - lnT;")
        for k, sp in enumerate(m.species):
            e(f"const double g{k} = {_g_expr(k, sp, f'lo_{int(sp.Tmid)}')};")

    e("// Molar production rates [mol/cm^3/s] from T and concentrations C [mol/cm^3].")
    e("__device__ __forceinline__ static void wdot(const double T, const double* __restrict__ C_, double* __restrict__ wdot_) {")
    e.ind += 1
    e("const double invT = 1.0 / T;")
    e("const double lnT = pgb_log(T);")
    for k in range(ns):
        e(f"const double C{k} = C_[{k}];")
    emit_gibbs()
    emit_rates_fp64(False)
    for k in range(ns):
        e(f"wdot_[{k}] = wd{k};")
    e.ind -= 1
    e("}")
    e()
    e("// Reactor RHS (constant-pressure RhoH): y = [rhoY_k (g/cm^3), T], F = rhoY forcing,")
    e("// Fh = rho h forcing. ydot_k = W_k wdot_k + F_k; dT/dt = (Fh - sum h_k ydot_k) / (rho cp).")
    e("__device__ __forceinline__ static void rhs(const double* __restrict__ y, const double* __restrict__ F, const double Fh, double* __restrict__ ydot) {")
    e.ind += 1
    e(f"const double T = y[{ns}];")
    e("const double invT = 1.0 / T;")
    e("const double lnT = pgb_log(T);")
    exact = kernel_family(m) == "thread"  # another kernel repeats the bits of this function
    for k in range(ns):
        c = _f(1.0 / W[k])
        e(f"const double C{k} = " + (f"__dmul_rn(y[{k}], {c});" if exact else f"y[{k}] * {c};"))
    emit_gibbs()
    if exact:
        emit_rates_exact()
    else:
        emit_rates_fp64(True)
    e("double hs = 0.0, rcp = 0.0;")
    for k, sp in enumerate(m.species):
        lf = f"lo_{int(sp.Tmid)}"
        e(f"{{ const double wm = fma(wd{k}, {_f(W[k])}, F[{k}]); ydot[{k}] = wm;")
        e(f"  hs = fma({_hW_expr(sp, lf, 1.0 / W[k])}, wm, hs);")
        e(f"  rcp = fma(y[{k}], {_cpW_expr(sp, lf, R_ERG / W[k])}, rcp); }}")
    e(f"ydot[{ns}] = fma(-hs, __dmul_rn({_f(R_ERG)}, T), Fh) / rcp;")
    e.ind -= 1
    e("}")
    e()
    # ---------------------------------------------------------------- Jacobian template
    e("// Analytic Jacobian d ydot / d y in arithmetic type R: entry (i, k) to A[i rs + k cs].")
    e("// Falloff blending factors are held frozen in the [M] and T derivatives. Every rounding is written")
    e("// out (fma, pgb_mul, pgb_add), so the kernels that inline it get the same bits.")
    e("template <class R>")
    e("__device__ __forceinline__ static void jac(const double* __restrict__ y, const double* __restrict__ Fd, const double Fhd, R* A, const int rs, const int cs) {")
    e.ind += 1
    mul = lambda *v: v[0] if len(v) == 1 else f"pgb_mul({mul(*v[:-1])}, {v[-1]})"
    add = lambda x, y_: f"pgb_add({x}, {y_})"
    neg = lambda x: x[1:] if x.startswith("-") else "-" + x
    fma = lambda x, y_, z: f"fma({x}, {y_}, {z})"

    def scaled(nu, x, acc):  # acc + nu x
        return add(acc, x if nu > 0 else neg(x)) if abs(nu) == 1 else fma(f"R({_f(nu)})", x, acc)

    e(f"const R T = (R)y[{ns}];")
    e("const R invT = R(1) / T;")
    e("const R lnT = pgb_logT<R>(T);")
    for k in range(ns):
        e(f"const R C{k} = (R)__dmul_rn(y[{k}], {_f(1.0 / W[k])});")
    # thermo in R
    tmids = sorted({s.Tmid for s in m.species})
    for t in tmids:
        e(f"const bool lo_{int(t)} = T < R({_f(t)});")
    for k, s in enumerate(m.species):
        for i in range(7):
            e(f"const R a{k}_{i} = lo_{int(s.Tmid)} ? R({_f(s.low[i])}) : R({_f(s.high[i])});")
    e("const R lnT1 = pgb_add(R(1), -lnT);")
    unused = {k for k in range(ns) if not any(m.species[k].name in r.reactants or m.species[k].name in r.products
                                              for r in m.reactions)}
    for k in range(ns):
        c = [f"a{k}_{i}" for i in range(7)]
        e(f"const R Ta{k} = {mul('T', c[4])};")
        g = fma(c[3], "R(-1.0 / 12.0)", mul(f"Ta{k}", "R(-0.05)"))
        g = fma("T", g, mul(c[2], "R(-1.0 / 6.0)"))
        g = fma("T", g, mul(c[1], "R(-0.5)"))
        g = fma(c[5], "invT", fma(c[0], "lnT1", mul("T", g)))
        e(f"const R g{k} = {g} - {c[6]};")
        h = fma(c[3], "R(0.25)", mul(f"Ta{k}", "R(0.2)"))
        h = fma(c[2], "R(1.0 / 3.0)", mul("T", h))
        h = fma(c[1], "R(0.5)", mul("T", h)) if k in unused else fma("T", h, mul(c[1], "R(0.5)"))
        e(f"const R h{k} = {fma(c[5], 'invT', fma('T', h, c[0]))};")
        e(f"const R cp{k} = {fma('T', fma('T', fma('T', add(c[3], f'Ta{k}'), c[2]), c[1]), c[0])};")
        d = fma("R(3)", c[3], mul("T", "R(4)", c[4]))
        e(f"const R dcp{k} = {fma('T', fma('R(2)', c[2], mul('T', d)), c[1])};")
    e("R J[N][N];")
    e("#pragma unroll")
    e("for (int i = 0; i < N; ++i)")
    e("#pragma unroll")
    e("  for (int k = 0; k < N; ++k) J[i][k] = R(0);")
    if any(r.kind != "elementary" for r in m.reactions):
        tot = "C0"
        for k in range(1, ns):
            tot = f"pgb_add_scaled<R>({tot}, y[{k}], {_f(1.0 / W[k])})" if k in total_only(m) else add(tot, f"C{k}")
        e(f"const R Ctot = {tot};")
    e(f"const R lnP0RT = pgb_add(R({_f(lnP0_R)}), -lnT);")
    for k in range(ns):
        e(f"R wd{k} = R(0);")
    for k in range(ns):
        e(f"R dT{k} = R(0);")
    for j, r in enumerate(m.reactions):
        e(f"// R{j}: {r.equation()}")
        e("{")
        e.ind += 1
        lnA = math.log(r.rate.A)
        ear = r.rate.Ea / R_CAL
        e(f"const R eT = {mul(f'R({_f(ear)})', 'invT')};")
        e(f"const R lnkf_inf = {add(fma(f'R({_f(r.rate.beta)})', 'lnT', '-eT'), f'R({_f(lnA)})')};")
        e(f"R dlnkf = {mul(add(f'R({_f(r.rate.beta)})', 'eT'), 'invT')};")
        if r.kind != "elementary":
            terms = "Ctot"
            for sname, eff in r.efficiencies.items():
                if eff != 1.0:
                    terms = fma(f"R({_f(eff - 1.0)})", f"C{idx[sname]}", terms)
            e(f"const R M = {terms};")
        if r.kind == "falloff":
            lnA0 = math.log(r.low.A)
            ear0 = r.low.Ea / R_CAL
            e(f"const R eT0 = {mul(f'R({_f(ear0)})', 'invT')};")
            e(f"const R lnk0 = {add(fma(f'R({_f(r.low.beta)})', 'lnT', '-eT0'), f'R({_f(lnA0)})')};")
            e(f"const R dlnk0 = {mul(add(f'R({_f(r.low.beta)})', 'eT0'), 'invT')};")
            e("const R k0 = pgb_expT<R>(lnk0);")
            e("const R kinf = pgb_expT<R>(lnkf_inf);")
            e("const R Pr = pgb_mul(M, pgb_expT<R>(lnk0 - lnkf_inf));")
            if r.troe:
                a, T3, T1 = r.troe[:3]
                fc = fma(f"R({_f(1.0 - a)})", f"pgb_expT<R>(T * R({_f(-1.0 / T3)}))",
                         mul(f"R({_f(a)})", f"pgb_expT<R>(T * R({_f(-1.0 / T1)}))"))
                if len(r.troe) > 3:
                    fc = add(fc, f"pgb_expT<R>(invT * R({_f(-r.troe[3])}))")
                e(f"const R lFc = {mul(f'pgb_logT<R>({fc})', f'R({_f(1.0 / LN10)})')};")
                e("const R cc = fma(R(-0.67), lFc, R(-0.4)), nn = fma(R(-1.27), lFc, R(0.75));")
                e(f"const R lPr = fma(pgb_logT<R>(Pr > R(1e-30) ? Pr : R(1e-30)), R({_f(1.0 / LN10)}), cc);")
                e("const R f1 = lPr / fma(R(-0.14), lPr, nn);")
                e(f"const R Fb = pgb_expT<R>({mul(f'R({_f(LN10)})', 'lFc')} / fma(f1, f1, R(1)));")
            else:
                e("const R Fb = R(1);")
            e("const R onePr = pgb_add(R(1), Pr);")
            e("const R kf = pgb_mul(pgb_mul(kinf, Pr) / onePr, Fb);")
            e("const R dkeff_dM = pgb_mul(Fb, k0) / pgb_mul(onePr, onePr);")
            e("dlnkf = pgb_add(dlnkf, (dlnk0 - dlnkf) / onePr);")
        else:
            e("const R kf = pgb_expT<R>(lnkf_inf);")
        pf_f = [idx[s] for s, nu in r.reactants.items() for _ in range(nu)]
        pr_f = [idx[s] for s, nu in r.products.items() for _ in range(nu)]
        e("const R Pf = " + mul(*[f"C{k}" for k in pf_f]) + ";")
        dnu = sum(r.products.values()) - sum(r.reactants.values())
        third = r.kind == "three_body"
        if r.reversible:
            e("const R Pp = " + mul(*[f"C{k}" for k in pr_f]) + ";")
            dg = dh = "R(0)"
            for side, sign in ((r.products, 1), (r.reactants, -1)):
                for s, nu in side.items():
                    dg = scaled(sign * nu, f"g{idx[s]}", dg)
                    dh = scaled(sign * nu, f"h{idx[s]}", dh)
            if dnu != 0:
                dg = scaled(-dnu, "lnP0RT", dg)
            e(f"const R kr = pgb_mul(kf, pgb_expT<R>(fmin({dg}, R(700))));")
            e(f"const R dlnkr = fma(-({dh} - R({dnu})), invT, dlnkf);")
            e("const R net = fma(kf, Pf, -pgb_mul(kr, Pp));")
            e(f"const R net_T = {fma(mul('kf', 'dlnkf'), 'Pf', neg(mul('kr', 'dlnkr', 'Pp')))};")
        else:
            e("const R net = pgb_mul(kf, Pf);")
            e(f"const R net_T = {mul('kf', 'dlnkf', 'Pf')};")
        # partials dq/dC_k, each a list of products
        dq: Dict[int, List[List[str]]] = {}

        def partials(side_list, coef):
            for k in sorted(set(side_list)):
                nu = side_list.count(k)
                others = list(side_list)
                others.remove(k)
                dq.setdefault(k, []).append(coef + ([f"R({nu})"] if nu > 1 else []) + [f"C{o}" for o in others])

        partials(pf_f, ["M", "kf"] if third else ["kf"])
        if r.reversible:
            partials(pr_f, ["-M", "kr"] if third else ["-kr"])
        if r.kind == "falloff":
            rev = "fma(-(kf > R(0) ? kr / kf : R(0)), Pp, Pf)" if r.reversible else "Pf"
            e(f"const R base = pgb_mul(dkeff_dM, {rev});")
        nus = {}
        for s, nu in r.reactants.items():
            nus[idx[s]] = nus.get(idx[s], 0) - nu
        for s, nu in r.products.items():
            nus[idx[s]] = nus.get(idx[s], 0) + nu
        nus = {i: nu for i, nu in nus.items() if nu != 0}
        # a product that is only ever added (coefficients 1 and -1) goes into the sums' multiply-adds
        whole = {k for k in dq if len(dq[k]) == 1 and len(dq[k][0]) > 1 and all(abs(nu * W[i] / W[k]) == 1.0
                                                                              for i, nu in nus.items())}
        for k, terms in dq.items():
            if k in whole:
                continue
            v = mul(*terms[0])
            for t in terms[1:]:
                v = fma(mul(*t[:-1]), t[-1], v) if len(t) > 1 else add(v, t[0])
            e(f"const R dq{k} = {v};")
        split = third and all(abs(nu) == 1 for nu in nus.values())
        if third and not split:
            e("const R q = pgb_mul(M, net), q_T = pgb_mul(M, net_T);")
        for i, nu in nus.items():
            for acc, v in ((f"wd{i}", "net"), (f"dT{i}", "net_T")):
                if split:
                    e(f"{acc} = {fma('M' if nu > 0 else '-M', v, acc)};")
                else:
                    e(f"{acc} = {scaled(nu, v.replace('net', 'q') if third else v, acc)};")
            for k in dq:
                co, at = nu * W[i] / W[k], f"J[{i}][{k}]"
                if k in whole:
                    t = dq[k][0]
                    e(f"{at} = {fma(mul(*t[:-1]) if co > 0 else neg(mul(*t[:-1])), t[-1], at)};")
                else:
                    e(f"{at} = {scaled(co, f'dq{k}', at)};")
            if r.kind != "elementary":
                effs = {idx[s]: eff for s, eff in r.efficiencies.items()}
                for k in range(ns):
                    eff = effs.get(k, 1.0)
                    if eff != 0.0:
                        e(f"J[{i}][{k}] = {scaled(nu * W[i] / W[k] * eff, 'net' if third else 'base', f'J[{i}][{k}]')};")
        e.ind -= 1
        e("}")
    # temperature column and energy row
    e("R Dm = R(0), dDm = R(0), Q = (R)Fhd;")
    for k in range(ns):
        e(f"const R wm{k} = fma(wd{k}, R({_f(W[k])}), (R)Fd[{k}]);")
        e(f"const R hm{k} = {mul(f'h{k}', f'R({_f(R_ERG / W[k])})', 'T')};")
        e(f"const R cpm{k} = {mul(f'cp{k}', f'R({_f(R_ERG / W[k])})')};")
        e(f"Dm = fma((R)y[{k}], cpm{k}, Dm);")
        e(f"dDm = fma({mul(f'(R)y[{k}]', f'dcp{k}')}, R({_f(R_ERG / W[k])}), dDm);")
        e(f"Q = fma(-hm{k}, wm{k}, Q);")
        e(f"J[{k}][{ns}] = {mul(f'R({_f(W[k])})', f'dT{k}')};")
    e("const R invD = R(1) / Dm;")
    e(f"const R QD2 = {mul('Q', 'invD', 'invD')};")
    for k in range(ns):
        sum_ = mul("hm0", f"J[0][{k}]") if ns == 1 else fma("hm0", f"J[0][{k}]", mul("hm1", f"J[1][{k}]"))
        for i in range(2, ns):
            sum_ = fma(f"hm{i}", f"J[{i}][{k}]", sum_)
        e(f"J[{ns}][{k}] = fma(-({sum_}), invD, -pgb_mul(QD2, cpm{k}));")
    sum_ = fma("cpm0", "wm0", mul("hm0", f"J[0][{ns}]"))
    for i in range(1, ns):
        sum_ = fma(f"hm{i}", f"J[{i}][{ns}]", fma(f"cpm{i}", f"wm{i}", sum_))
    e(f"J[{ns}][{ns}] = fma(-({sum_}), invD, -pgb_mul(QD2, dDm));")
    e("#pragma unroll")
    e("for (int i = 0; i < N; ++i)")
    e("#pragma unroll")
    e("  for (int k = 0; k < N; ++k) A[i * rs + k * cs] = J[i][k];")
    e.ind -= 1
    e("}")
    e.ind -= 1
    e("};")
    e("}  // namespace pgb")
    e(f"#endif  // {guard}")
    return e.text()


def main(outdir: str, names=("lidryer_syn", "drm19_syn", "gri_syn")):
    from ..workloads import load_mechanism
    os.makedirs(outdir, exist_ok=True)
    for n in names:
        m = load_mechanism(n)
        text = gen_header(m)
        path = os.path.join(outdir, f"mech_{n}.cuh")
        if os.path.exists(path):
            with open(path) as f:
                if f.read() == text:
                    continue  # unchanged: keep the timestamp so the library is not rebuilt
        with open(path, "w") as f:
            f.write(text)


if __name__ == "__main__":
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    main(sys.argv[1] if len(sys.argv) > 1 else os.path.join(here, "..", "csrc", "gen"))


# ---------------------------------------------------------------------------- tables
def rx_packed(rx, ns: int) -> list:
    """The four words of each reaction's TabRxPk record (mech_tables.cuh): x = kind | rev << 2 |
    nr << 3 | np << 5 | (dnu + 8) << 7 | (tb + 1) << 11 | (troe + 1) << 22; y, z = the reactant and
    product species slots, 10 bits each; w = 0."""
    assert ns <= 1024, "species index fields of the packed reaction record are 10 bits"
    out = []
    for (_, _, _, kind, rev, rs, ps, dnu, tb, tr) in rx:
        assert -8 <= dnu <= 7 and tb + 1 < 2048 and tr + 1 < 1024
        x = kind | rev << 2 | len(rs) << 3 | len(ps) << 5 | (dnu + 8) << 7 | (tb + 1) << 11 | (tr + 1) << 22
        y = sum(k << (10 * s_) for s_, k in enumerate(rs))
        z = sum(k << (10 * s_) for s_, k in enumerate(ps))
        out.append((x, y, z, 0))
    return out


def _f32(x: float) -> float:
    return struct.unpack("f", struct.pack("f", x))[0]


def enthalpy_about(a, W: float, tref: float) -> list:
    """h/R per gram of NASA-7 coefficients `a` as a polynomial in x = T - tref, [d1..d5, d0] with
    h = d0 + x (d1 + x (d2 + ...)); each rounded once."""
    t, w = Fraction(tref), Fraction(W)
    cp = [Fraction(v) / w for v in a[:5]]
    d = [sum(cp[j] * math.comb(j, i) * t ** (j - i) for j in range(i, 5)) / (i + 1) for i in range(5)]
    d0 = Fraction(a[5]) / w + sum(cp[i] * t ** (i + 1) / (i + 1) for i in range(5))
    return [float(v) for v in d] + [float(d0)]


def jac_stream(m: Mechanism, rx, tb_rows, codes, neg, T: int, LDA: int, L: int = 32):
    """The contribution program (kJacC, kJacNeg) in the form the kernels stream: (quads, entries,
    x0, nx).

    quads[q][lane] holds the lane's terms 4q..4q+3, one word each: bits 0-12 the index of the term's
    first partial (8 j + slot of reaction j, or 8 NR + x for partial x below), 13-19 further slots
    1..7 of the same reaction to add, 20 the sign of the coefficient (1: minus), 21 last term of its
    entry, 22 the collider slot is scaled by its efficiency, 23 T column (added even when 0).
    entries[e][lane] = (|c| in FP64, |c| in FP32, i LDA + k) of the lane's e-th entry.
    Partials 8 NR + x0[tb] + s: the [M] partial of third-body row tb times the efficiency of its
    s-th listed collider, so a collider term needs no efficiency of its own."""
    ns = m.ns
    x0, nx = [], 0
    for effs in tb_rows:
        x0.append(nx)
        nx += len(effs)
    n_rx = len(rx)
    assert 8 * n_rx + nx <= 8192, "partial index field too narrow for this mechanism"
    nq = (T + 3) // 4
    quads = [[[0, 0, 0, 0] for _ in range(L)] for _ in range(nq)]
    ents = [[] for _ in range(L)]
    W = [s.W for s in m.species]
    for l_ in range(L):
        for t in range(T):
            c = codes[L * t + l_]
            if c == 0:
                continue  # padding: adds to a sum that is never stored
            j, tg = c & 0x1FF, (c >> 9) & 0xFFF
            i, k = divmod(tg, LDA)
            word = ((neg[t] >> l_) & 1) << 20 | ((c >> 29) & 1) << 21
            if c & (1 << 21):
                word |= (8 * j) | 1 << 23
            else:
                slots = [1 + b for b in range(6) if c & (1 << (22 + b))] + ([7] if c & (1 << 28) else [])
                scaled = bool(c & (1 << 31))
                if slots == [7] and scaled:
                    tb = rx[j][8]
                    word |= 8 * n_rx + x0[tb] + [sp for sp, _ in tb_rows[tb]].index(k)
                else:
                    word |= 8 * j + slots[0]
                    for s_ in slots[1:]:
                        word |= 1 << (12 + s_)
                    if scaled:
                        word |= 1 << 22
            quads[t // 4][l_][t % 4] = word
            if c & (1 << 30):
                wd = W[i] if k == ns else W[i] * (1.0 / W[k])
                wf = _f32(W[i]) if k == ns else _f32(_f32(W[i]) * _f32(1.0 / W[k]))
                ents[l_].append((wd, wf, tg))
    return quads, ents, x0, nx


def deal_program(ents, L: int, LDA: int):
    """The program's entries dealt to L lanes, largest first, to the lane with the fewest terms so far:
    (terms per lane, codes, sign planes), term t of lane l at L t + l."""
    lanes = [[] for _ in range(L)]
    load = [0] * L
    for key, terms in ents:
        l_ = min(range(L), key=lambda v: (load[v], v))
        lanes[l_].append((key, terms))
        load[l_] += len(terms)
    T = max(load)
    codes, neg = [0] * (L * T), [0] * T
    for l_ in range(L):
        t = 0
        for (i, k), terms in lanes[l_]:
            for n_, (code, isr, _) in enumerate(terms):
                flags = ((1 << 29) if n_ == len(terms) - 1 else 0) | ((1 << 30) if n_ == 0 else 0)
                codes[L * t + l_] = (code | ((i * LDA + k) << 9) | flags) & 0xFFFFFFFF
                neg[t] |= int(isr) << l_
                t += 1
    return T, codes, neg


def emit_team_stream(e: _Emitter, qual: str, m: Mechanism, rx, tb_rows, ents, LDA: int, L: int = 128):
    """The program once more, for the L lanes of a team of warps."""
    T, codes, neg = deal_program(ents, L, LDA)
    quads, lane_ents, _, _ = jac_stream(m, rx, tb_rows, codes, neg, T, LDA, L)
    ne = max(len(v) for v in lane_ents) + 1
    e(f"constexpr int NJQT = {len(quads)}, NJET = {ne};")
    e(f"{qual} uint4 kJacQT[{L} * NJQT] = {{")
    for q in quads:
        e("  " + ", ".join("{" + ", ".join(f"{w}u" for w in lane) + "}" for lane in q) + ",")
    e("};")
    for R, suf, col in (("double", "D", 0), ("float", "F", 1)):
        e(f"{qual} TabJacEnt<{R}> kJacEntT{suf}[{L} * NJET] = {{")
        for n_ in range(ne):
            row = [v[n_] if n_ < len(v) else (0.0, 0.0, 0) for v in lane_ents]
            e("  " + ", ".join("{" + _f(v[col]) + ("f" if col else "") + f", {v[2]}}}" for v in row) + ",")
        e("};")


def emit_jac_stream(e: _Emitter, qual: str, m: Mechanism, rx, tb_rows, codes, neg, T: int, LDA: int):
    quads, ents, x0, nx = jac_stream(m, rx, tb_rows, codes, neg, T, LDA)
    ne = max(len(v) for v in ents) + 1  # one past the end: read ahead, never used
    e(f"constexpr int NJQ = {len(quads)}, NJE = {ne}, NJX = {nx};  // quads, entries per lane; scaled partials")
    e(f"{qual} uint4 kJacQ[32 * NJQ] = {{")
    for q in quads:
        e("  " + ", ".join("{" + ", ".join(f"{w}u" for w in lane) + "}" for lane in q) + ",")
    e("};")
    for R, suf, col in (("double", "D", 0), ("float", "F", 1)):
        e(f"{qual} TabJacEnt<{R}> kJacEnt{suf}[32 * NJE] = {{")
        for n_ in range(ne):
            row = [v[n_] if n_ < len(v) else (0.0, 0.0, 0) for v in ents]
            e("  " + ", ".join("{" + _f(v[col]) + ("f" if col else "") + f", {v[2]}}}" for v in row) + ",")
        e("};")
    e(f"{qual} int kJacX0[NTB] = {{{', '.join(str(8 * len(rx) + v) for v in (x0 or [0]))}}};")


def emit_unrolled_order(e: _Emitter, qual: str, m: Mechanism, order):
    """What a lane-parallel evaluation needs to repeat the unrolled right-hand side (gen_header,
    emit_rates_exact): the constants as that code folds them, and each species' reactions in the order
    in which it adds them (input order; values are positions in `order`)."""
    e(f"{qual} TabUnrolled kUnrolled[NS] = {{")
    for s in m.species:
        rows = []
        for a in (s.low, s.high):
            rows.append([a[0] * 1.0, a[1] * -0.5, a[2] * (-1.0 / 6.0), a[3] * (-1.0 / 12.0), a[4] * -0.05, a[5] * 1.0,
                         a[6] * -1.0])
        for a in (s.low, s.high):
            w = 1.0 / s.W
            rows.append([a[0] * 1.0 * w, a[1] * 0.5 * w, a[2] * (1.0 / 3.0) * w, a[3] * 0.25 * w, a[4] * 0.2 * w,
                         a[5] * 1.0 * w])
        for a in (s.low, s.high):
            w = R_ERG / s.W
            rows.append([a[i] * w for i in range(5)])
        e(f"  {{{_f(1.0 / s.W)}, {_f(s.W)}, {_f(s.Tmid)}, {int(m.index(s.name) in total_only(m))}, "
          + ", ".join("{" + ", ".join(_f(v) for v in r) + "}" for r in rows) + "},")
    e("};")
    pos = {j: i for i, j in enumerate(order)}
    off, jj, nu, tb = [0], [], [], []
    for s in m.species:
        for j, r in enumerate(m.reactions):
            net = r.products.get(s.name, 0) - r.reactants.get(s.name, 0)
            if net != 0:
                jj.append(pos[j])
                nu.append(float(net))
                tb.append(int(abs(net) == 1 and j == fused_third_body(m)))
        off.append(len(jj))
    e(f"{qual} int kUnM[{len(jj)}] = {{{', '.join(str(v) for v in tb)}}};")
    e(f"{qual} int kUnOff[NS + 1] = {{{', '.join(str(v) for v in off)}}};")
    e(f"{qual} int kUnJ[{len(jj)}] = {{{', '.join(str(v) for v in jj)}}};")
    e(f"{qual} double kUnNu[{len(jj)}] = {{{', '.join(_f(v) for v in nu)}}};")


def gen_tables(m: Mechanism, space: str = "constant") -> str:
    """Mechanism tables for the table-driven kernels: per-species W, NASA-7 sets, per-reaction
    Arrhenius data, stoichiometry as species slots (a species with coefficient 2 occupies two
    slots), sparse third-body efficiencies and Troe parameters.

    space "constant": __constant__ arrays in namespace tab_<name> (per-thread kernels: every lane
    reads the same entry, a constant-cache broadcast). space "global": read-only global arrays in
    namespace tabg_<name> (warp-per-cell kernels: lanes read different entries through L1; also
    the only choice when the tables exceed the 64 KB constant bank), plus the species-major list
    of the reactions each species takes part in with its net coefficient (production rates as a
    gather)."""
    check_supported(m)
    glob = space == "global"
    qual = "__device__ const" if glob else "__device__ __constant__"
    nsname = f"tabg_{m.name}" if glob else f"tab_{m.name}"
    ns = m.ns
    idx = {s.name: i for i, s in enumerate(m.species)}
    tb_rows, troe_rows = [], []
    rx = []
    for r in m.reactions:
        rs = [idx[s] for s, nu in r.reactants.items() for _ in range(nu)]
        ps = [idx[s] for s, nu in r.products.items() for _ in range(nu)]
        assert len(rs) <= 3 and len(ps) <= 3
        kind = {"elementary": 0, "three_body": 1, "falloff": 2}[r.kind]
        tb = -1
        if r.kind != "elementary":
            tb = len(tb_rows)
            effs = [(idx[s], e - 1.0) for s, e in r.efficiencies.items() if e != 1.0]
            tb_rows.append(effs)
        tr = -1
        if r.kind == "falloff":
            tr = len(troe_rows)
            lnA0 = math.log(r.low.A)
            t = r.troe or []
            troe_rows.append((lnA0, r.low.beta, -r.low.Ea / R_CAL, len(t),
                              (1.0 - t[0]) if t else 0.0, (-1.0 / t[1]) if t else 0.0,
                              t[0] if t else 0.0, (-1.0 / t[2]) if t else 0.0,
                              (-t[3]) if len(t) > 3 else 0.0))
        dnu = sum(r.products.values()) - sum(r.reactants.values())
        rx.append((math.log(r.rate.A), r.rate.beta, -r.rate.Ea / R_CAL, kind, int(r.reversible),
                   rs, ps, dnu, tb, tr))
    if glob:
        # warp-per-cell kernels give consecutive reactions to the lanes of a warp: group them by
        # kind (elementary, third-body, falloff) so a 32-reaction pass rarely mixes code paths
        order = sorted(range(len(rx)), key=lambda j: (rx[j][3], j))
        rx = [rx[j] for j in order]
    maxeff = max([len(t) for t in tb_rows] + [1])
    tmids = sorted({s.Tmid for s in m.species})
    # where the mixture's enthalpy polynomial is expanded: mid-range below and above a common Tmid
    # (errors of T from rho h against 64 bits on the workloads' states, 2-norm: expanded about 0 K 1.0 to
    # 1.4e-16, about 1000 K 0.7 to 1.1e-16, so 0.6 to 0.8e-16), else one point, as ranges mix
    tref = (600.0, 1800.0) if len(tmids) == 1 else (1000.0, 1000.0)
    e = _Emitter()
    e(f"// GENERATED by pelelm_gb300/mech/codegen.py (tables, {space} memory) from pelelm_gb300/data/{m.name}.json.")
    guard = f"PGB_{nsname.upper()}_CUH"
    e(f"#ifndef {guard}")
    e(f"#define {guard}")
    e('#include "../mech_tables.cuh"')
    e("namespace pgb {")
    e(f"namespace {nsname} {{")
    e(f"constexpr int NS = {ns}, NR = {m.nr}, NTB = {max(1, len(tb_rows))}, NTROE = {max(1, len(troe_rows))}, MAXEFF = {maxeff};")
    for R, suf, cast in (("double", "D", lambda x: _f(x)), ("float", "F", lambda x: _f(x) + "f")):
        e(f"{qual} TabSpecies<{R}> kSpecies{suf}[NS] = {{")
        def gco(a):
            return [a[0], -a[1] / 2, -a[2] / 6, -a[3] / 12, -a[4] / 20, a[5], -a[6]]

        def hco(a):
            return [a[0], a[1] / 2, a[2] / 3, a[3] / 4, a[4] / 5, a[5]]

        for sp_ in m.species:
            arrs = [sp_.low, sp_.high, gco(sp_.low), gco(sp_.high), hco(sp_.low), hco(sp_.high),
                    [v / sp_.W for v in hco(sp_.low)], [v / sp_.W for v in hco(sp_.high)]]
            body = ", ".join("{" + ", ".join(cast(a_) for a_ in arr) + "}" for arr in arrs)
            e(f"  {{{cast(sp_.W)}, {cast(1.0 / sp_.W)}, {cast(sp_.Tmid)}, {body}}},")
        e("};")
        e(f"{qual} TabReaction<{R}> kReactions{suf}[NR] = {{")
        for (lnA, beta, mear, kind, rev, rs, ps, dnu, tb, tr) in rx:
            rsl = ", ".join(str(x) for x in (rs + [0, 0, 0])[:3])
            psl = ", ".join(str(x) for x in (ps + [0, 0, 0])[:3])
            e(f"  {{{cast(lnA)}, {cast(beta)}, {cast(mear)}, {kind}, {rev}, {len(rs)}, {len(ps)}, {{{rsl}}}, {{{psl}}}, {dnu}, {tb}, {tr}}},")
        e("};")
        e(f"{qual} TabThirdBody<{R}> kThirdBody{suf}[NTB] = {{")
        if not tb_rows:
            e(f"  {{0, {{0}}, {{{cast(0.0)}}}}},")
        for effs in tb_rows:
            sp = ", ".join(str(k) for k, _ in effs) or "0"
            ev = ", ".join(cast(v) for _, v in effs) or cast(0.0)
            e(f"  {{{len(effs)}, {{{sp}}}, {{{ev}}}}},")
        e("};")
        e(f"{qual} TabTroe<{R}> kTroe{suf}[NTROE] = {{")
        if not troe_rows:
            e("  {" + ", ".join([cast(0.0)] * 3 + ["0"] + [cast(0.0)] * 5) + "},")
        for t in troe_rows:
            e("  {" + ", ".join(cast(v) if isinstance(v, float) else str(v) for v in t) + "},")
        e("};")
    if glob:
        # species-major reaction lists: species k takes part in reactions kSpRxJ[kSpRxOff[k]..
        # kSpRxOff[k+1]) with net molar coefficient kSpRxNu (products minus reactants), in
        # reaction order
        off, jj, nu = [0], [], []
        for k in range(ns):
            for j, (_, _, _, _, _, rs_, ps_, _, _, _) in enumerate(rx):
                net = ps_.count(k) - rs_.count(k)
                if net != 0:
                    jj.append(j)
                    nu.append(float(net))
            off.append(len(jj))
        # Jacobian contribution program of the cooperative setup (warp and lane-group kernels):
        # every nonzero species entry A[i][k] (and T-column entry A[i][NS]) of the analytic
        # Jacobian with its ordered terms. A term of reaction j adds c * v to its entry, c =
        # -+W_i / W_k (-+W_i in the T column; minus for a reactant row slot) and v the sum of the
        # stored partials of j that its code selects. Terms keep the order of the reaction walk
        # they replace: reactions ascending, then the row slots of the reaction. Entries go to
        # the 32 lanes largest first, to the lane with the fewest terms so far; each lane's terms
        # are interleaved (term t of lane l at 32 t + l, lanes padded with empty terms to the
        # longest). The kernels read it in the form that jac_stream makes of it.
        # code bits: 0-8 reaction (table order), 9-20 entry i * (N + 1) + k, 21 dq/dT (T column),
        # 22-24 / 25-27 the reactant / product slots of j holding species k, 28 the collider
        # term dq/d[M] times the efficiency of k, 29 last term of its entry (store the sum), 30
        # first term of its entry, 31 efficiency different from 1 (read it); the sign of c is
        # carried by bit 29 of a separate bit plane (kJacNeg, one bit per term).
        N = ns + 1
        LDA = N + 1
        assert m.nr <= 512 and N * LDA <= 4096, "program code fields too narrow for this mechanism"
        prog = {}
        for j, (_, _, _, kind_, _, rs_, ps_, _, tb_, _) in enumerate(rx):
            effs = dict(tb_rows[tb_]) if kind_ != 0 else {}
            rows = [(i, True) for i in rs_] + [(i, False) for i in ps_]
            cols = sorted(set(rs_) | set(ps_)) if kind_ == 0 else list(range(ns))
            for k in cols:
                code = j
                for s_, sk in enumerate(rs_):
                    if sk == k:
                        code |= 1 << (22 + s_)
                for s_, sk in enumerate(ps_):
                    if sk == k:
                        code |= 1 << (25 + s_)
                em1 = None
                if kind_ != 0:
                    code |= 1 << 28
                    em1 = effs.get(k)
                    if em1 is not None:
                        code |= 1 << 31
                for (i, isr) in rows:
                    prog.setdefault((i, k), []).append((code, isr, em1))
            for (i, isr) in rows:
                prog.setdefault((i, ns), []).append((j | (1 << 21), isr, None))
        ents = sorted(prog.items(), key=lambda kv: (-len(kv[1]), kv[0]))
        lanes = [[] for _ in range(32)]
        load = [0] * 32
        for key, terms in ents:
            l_ = min(range(32), key=lambda x: (load[x], x))
            lanes[l_].append((key, terms))
            load[l_] += len(terms)
        T = max(load)
        codes = [0] * (32 * T)
        neg = [0] * T  # bit l of word t: term t of lane l has a reactant row slot (c < 0)
        effD = ["1.0"] * (32 * T)
        effF = ["1.0f"] * (32 * T)
        for l_ in range(32):
            t = 0
            for (i, k), terms in lanes[l_]:
                for n_, (code, isr, em1) in enumerate(terms):
                    pos = 32 * t + l_
                    flags = ((1 << 29) if n_ == len(terms) - 1 else 0) | ((1 << 30) if n_ == 0 else 0)
                    codes[pos] = (code | ((i * LDA + k) << 9) | flags) & 0xFFFFFFFF
                    if isr:
                        neg[t] |= 1 << l_
                    if em1 is not None:
                        effD[pos] = f"(1.0 + {_f(em1)})"
                        effF[pos] = f"(1.0f + {_f(em1)}f)"
                    t += 1
        e(f"constexpr int NJT = {T};  // program terms per lane (padded)")
        e("#if 0  // the program that the streamed form below is made from: no kernel reads it")
        e(f"{qual} unsigned kJacC[32 * NJT] = {{{', '.join(str(x) + 'u' for x in codes)}}};")
        e(f"{qual} unsigned kJacNeg[NJT] = {{{', '.join(str(x) + 'u' for x in neg)}}};")
        e("#endif")
        e(f"{qual} double kJacEffD[32 * NJT] = {{{', '.join(effD)}}};")
        e(f"{qual} float kJacEffF[32 * NJT] = {{{', '.join(effF)}}};")
        emit_jac_stream(e, qual, m, rx, tb_rows, codes, neg, T, LDA)
        if kernel_family(m) == "warp":
            emit_team_stream(e, qual, m, rx, tb_rows, ents, LDA)
        # packed reaction records of the FP64 rate of progress (TabRxArr / TabRxPk)
        e(f"{qual} TabRxArr kRxArr[NR] = {{")
        for (lnA, beta, mear, *_r) in rx:
            e(f"  {{{_f(lnA)}, {_f(beta)}, {_f(mear)}, 0.0}},")
        e("};")
        e(f"{qual} TabRxPk kRxPk[NR] = {{")
        for w in rx_packed(rx, ns):
            e("  {" + ", ".join(f"{v}u" for v in w) + "},")
        e("};")
        if kernel_family(m) == "thread":
            emit_unrolled_order(e, qual, m, order)
        lens = [off[k + 1] - off[k] for k in range(ns)]
        by_len = sorted(range(ns), key=lambda k: (-lens[k], k))
        e(f"constexpr int NSPRX = {len(jj)};")
        e(f"{qual} int kSpByLen[NS] = {{{', '.join(str(k) for k in by_len)}}};  // longest lists first")
        e(f"{qual} int kSpRxOff[NS + 1] = {{{', '.join(str(x) for x in off)}}};")
        e(f"{qual} int kSpRxJ[NSPRX] = {{{', '.join(str(x) for x in jj)}}};")
        e(f"{qual} double kSpRxNu[NSPRX] = {{{', '.join(_f(x) for x in nu)}}};")
    hmid = []  # h/R per gram of every species at the common Tmid (low-range polynomial)
    joined = len(tmids) == 1  # every h continuous there, but for rounding
    for s in m.species:
        t = tmids[0]
        lo, hi = (a[5] + t * (a[0] + t * (a[1] / 2 + t * (a[2] / 3 + t * (a[3] / 4 + t * a[4] / 5)))) for a in (s.low, s.high))
        joined = joined and abs(lo - hi) <= 1e-12 * (abs(lo) + t)
        hmid.append(lo / s.W)
    e(f"{qual} TabEnthalpy kEnthalpy[NS] = {{")
    for s in m.species:
        e("  {" + ", ".join("{" + ", ".join(_f(v) for v in enthalpy_about(a, s.W, t)) + "}"
                            for a, t in zip((s.low, s.high), tref)) + "},")
    e("};")
    e(f"{qual} double kHMid[NS] = {{{', '.join(_f(v) for v in hmid)}}};")
    e("struct Tables {")
    e(f"  static constexpr double TMID = {_f(tmids[0]) if len(tmids) == 1 else '-1.0'};  // common Tmid, or -1")
    e(f"  static constexpr double TREF_LO = {_f(tref[0])}, TREF_HI = {_f(tref[1])};  // of the mixture polynomial")
    e(f"  static constexpr bool JOINED = {'true' if joined else 'false'};  // no jump of any h at that Tmid")
    e("  __device__ static const TabEnthalpy& enthalpy(int k) { return kEnthalpy[k]; }")
    e("  __device__ static double h_mid(int k) { return kHMid[k]; }")
    e(f"  static constexpr int NS = {ns}, NR = {m.nr};")
    if glob:
        if kernel_family(m) == "thread":
            e("  __device__ static const TabUnrolled& un(int k) { return kUnrolled[k]; }")
            e("  __device__ static int un_begin(int k) { return kUnOff[k]; }")
            e("  __device__ static int un_j(int e) { return kUnJ[e]; }")
            e("  __device__ static bool un_m(int e) { return kUnM[e] != 0; }  // q [M] is fused here")
            e("  __device__ static double un_nu(int e) { return kUnNu[e]; }")
        e("  __device__ static int sprx_begin(int k) { return kSpRxOff[k]; }")
        e(f"  static constexpr int MAXR = {max(len(r[5]) for r in rx)}, MAXP = {max(len(r[6]) for r in rx)};  // slots a side")
        e("  __device__ static int sprx_by_len(int i) { return kSpByLen[i]; }")
        e("  __device__ static int sprx_end(int k) { return kSpRxOff[k + 1]; }")
        e("  __device__ static int sprx_j(int e) { return kSpRxJ[e]; }")
        e("  __device__ static double sprx_nu(int e) { return kSpRxNu[e]; }")
        e("  __device__ static const TabRxArr& rx_arr(int j) { return kRxArr[j]; }")
        e("  __device__ static TabRxPk rx_pk(int j) { return kRxPk[j]; }")
        e("  static constexpr int JAC_QUADS = NJQ, JAC_ENTS = NJE, JAC_X = NJX;")
        e("  __device__ static uint4 jac_quad(int c) { return kJacQ[c]; }")
        e("  template <class R> __device__ static const TabJacEnt<R>& jac_ent(int c) {")
        e("    if constexpr (sizeof(R) == sizeof(double)) return kJacEntD[c]; else return kJacEntF[c];")
        e("  }")
        e("  __device__ static int jac_x0(int tb) { return kJacX0[tb]; }")
        if kernel_family(m) == "warp":
            e("  static constexpr int TEAM_QUADS = NJQT, TEAM_ENTS = NJET;")
            e("  __device__ static uint4 team_quad(int c) { return kJacQT[c]; }")
            e("  template <class R> __device__ static const TabJacEnt<R>& team_ent(int c) {")
            e("    if constexpr (sizeof(R) == sizeof(double)) return kJacEntTD[c]; else return kJacEntTF[c];")
            e("  }")
        e("  template <class R> __device__ static R jac_eff(int c) {")
        e("    if constexpr (sizeof(R) == sizeof(double)) return kJacEffD[c]; else return kJacEffF[c];")
        e("  }")
    for nm, typ, arr in (("sp", "TabSpecies", "kSpecies"), ("rx", "TabReaction", "kReactions"),
                         ("tb", "TabThirdBody", "kThirdBody"), ("troe", "TabTroe", "kTroe")):
        e(f"  template <class R> __device__ static const {typ}<R>& {nm}(int i) {{")
        e(f"    if constexpr (sizeof(R) == sizeof(double)) return {arr}D[i]; else return {arr}F[i];")
        e("  }")
    e("};")
    e(f"}}  // namespace {nsname}")
    e("}  // namespace pgb")
    e(f"#endif  // {guard}")
    return e.text()


def kernel_family(m: Mechanism) -> str:
    """Which persistent BDF kernels a mechanism gets: "thread" (cell per thread and per warp)
    up to 12 species, "group" (cell per thread, per lane group and per warp) while the ODE size
    stays within one warp's lanes (N <= 32), else "warp" only (one cell's state no longer fits a
    thread)."""
    if m.ns <= 12:
        return "thread"
    return "group" if m.ns + 1 <= 32 else "warp"


def constant_tables(m: Mechanism) -> bool:
    """Tables in the 64 KB constant bank for the per-thread kernels (mechanisms that have them);
    every mechanism also gets the global-memory tables of the lane-group and warp kernels."""
    return kernel_family(m) != "warp"


def write_tables(outdir: str, names=("lidryer_syn", "drm19_syn", "gri_syn")):
    from ..workloads import load_mechanism
    for n in names:
        m = load_mechanism(n)
        outs = [(f"tabg_{n}.cuh", gen_tables(m, "global"))]
        if constant_tables(m):
            outs.append((f"tab_{n}.cuh", gen_tables(m, "constant")))
        for fname, text in outs:
            path = os.path.join(outdir, fname)
            if os.path.exists(path):
                with open(path) as f:
                    if f.read() == text:
                        continue
            with open(path, "w") as f:
                f.write(text)


# ---------------------------------------------------------------------------- registry
_ENTRY_MACRO = {"thread": "PGB_MECH_ENTRY", "group": "PGB_MECH_ENTRY_GROUP", "warp": "PGB_MECH_ENTRY_WARP"}


def write_units(outdir: str, names) -> list:
    """One translation unit per mechanism (its kernels and registry entry) and the registry list
    included by csrc/reactor.cu; returns the unit paths. Files are rewritten only on change."""
    from ..workloads import load_mechanism

    def put(path, text):
        if os.path.exists(path):
            with open(path) as f:
                if f.read() == text:
                    return
        with open(path, "w") as f:
            f.write(text)

    units = []
    reg = ["// GENERATED by pelelm_gb300/mech/codegen.py from the mechanisms in pelelm_gb300/data/.",
           "// Registry of the compiled mechanisms (one unit_<name>.cu each), included by reactor.cu.",
           "namespace pgb_host {"]
    for n in names:
        m = load_mechanism(n)
        fam = kernel_family(m)
        text = "\n".join([
            f"// GENERATED by pelelm_gb300/mech/codegen.py from pelelm_gb300/data/{n}.json.",
            f"// Kernels of mechanism {n} ({m.ns} species, {m.nr} reactions; BDF kernel family: {fam}) and",
            "// its registry entry.",
            f'#include "mech_{n}.cuh"',
            '#include "../reactor_registry.cuh"',
            "",
            "namespace pgb_host {",
            f"extern const MechEntry kEntry_{n} = {_ENTRY_MACRO[fam]}(pgb::Mech_{n});",
            "}  // namespace pgb_host",
            ""])
        path = os.path.join(outdir, f"unit_{n}.cu")
        put(path, text)
        units.append(path)
        reg.append(f"extern const MechEntry kEntry_{n};")
    reg.append("}  // namespace pgb_host")
    reg.append("#define PGB_MECH_LIST " + ", ".join(f"&::pgb_host::kEntry_{n}" for n in names))
    put(os.path.join(outdir, "mech_registry.inc"), "\n".join(reg) + "\n")
    return units
