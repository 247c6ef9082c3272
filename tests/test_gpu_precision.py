"""T from rho h against extended precision."""
import numpy as np
import pytest

from pelelm_gb300.reactor import rhoh_to_temp
from pelelm_gb300.workloads import CONFIGS, load_mechanism, make_cells

R_ERG = 8.31446261815324e7


@pytest.mark.gpu
@pytest.mark.parametrize("cfgname", ["lidryer_amr120", "drm19_2M", "gri_1M"])
def test_temperature_is_within_twice_its_own_rounding(native_lib, cuda, cfgname):
    """2-norm of the error over all cells: T as a double is off by one rounding, the result of the sums,
    polynomials and the last Newton step by at most as much again."""
    torch = cuda
    cfg = CONFIGS[cfgname]
    m, n = load_mechanism(cfg.mech), 4096
    cs = make_cells(cfg, n, seed=4)
    rY = cs.rY * 1e3
    rE = cs.rE * 0.1 + rY.sum(1) * 4e4 * np.random.default_rng(1).uniform(-0.5, 0.5, n)
    ld = np.longdouble
    lo, hi = (np.array([getattr(s, q) for s in m.species]).astype(ld) for q in ("low", "high"))
    W, Tmid = (np.array([getattr(s, q) for s in m.species]).astype(ld) for q in ("W", "Tmid"))
    rho = rY.astype(ld).sum(1)
    Y, h, T = rY.astype(ld) / rho[:, None], rE.astype(ld) / rho * ld(10) ** 4, cs.T.astype(ld)
    for _ in range(12):
        t = T[:, None]
        a = np.where((t < Tmid)[:, :, None], lo[None], hi[None])
        hk = a[..., 5] + t * (a[..., 0] + t * (a[..., 1] / 2 + t * (a[..., 2] / 3 + t * (a[..., 3] / 4 + t * a[..., 4] / 5))))
        ck = a[..., 0] + t * (a[..., 1] + t * (a[..., 2] + t * (a[..., 3] + t * a[..., 4])))
        dT = (h - (Y * hk * ld(R_ERG) / W).sum(1)) / (Y * ck * ld(R_ERG) / W).sum(1)
        T = T + np.clip(dT, -100, 100)
    assert np.abs(dT).max() < 1e-14 * float(T.max())

    def t3(v, nc):
        return torch.tensor(np.ascontiguousarray(np.asarray(v).reshape(n, nc).T.reshape(nc, 1, 1, n)), device="cuda")

    Tg = t3(cs.T, 1)
    rhoh_to_temp(cfg.mech, ((0, 0, 0), (n - 1, 0, 0)), t3(rY, m.ns), t3(rE, 1), Tg)
    got = Tg.cpu().numpy().reshape(n).astype(ld)

    def off(x):
        return float(np.sqrt(((x - T) ** 2).sum() / (T ** 2).sum()))

    assert off(got) <= 2.0 * off(T.astype(np.float64).astype(ld)), (off(got), off(T.astype(np.float64).astype(ld)))


@pytest.mark.gpu
@pytest.mark.parametrize("tmax", [5000.0, 8000.0])
def test_cells_without_mass_end_where_the_iteration_stops(native_lib, cuda, tmax):
    """No mass, no energy: 50 steps of +100 K, up to the limit (as before there were mixture sums)."""
    torch = cuda
    n, ns = 8, 9
    z = dict(device="cuda", dtype=torch.float64)
    for e in (0.0, 5.0, -5.0):
        T = torch.full((1, 1, 1, n), 300.0, **z)
        rhoh_to_temp("lidryer_syn", ((0, 0, 0), (n - 1, 0, 0)), torch.zeros(ns, 1, 1, n, **z), torch.full((1, 1, 1, n), e, **z), T,
                     tmax=tmax)
        assert torch.all(T == min(tmax, 5300.0)), (e, T)


@pytest.mark.gpu
@pytest.mark.parametrize("cfgname,bound", [("lidryer_amr120", 2.9e-15), ("drm19_2M", 4.2e-15)])
def test_reaction_rates_against_extended_precision(native_lib, cuda, cfgname, bound):
    """2-norm over cells and species of the error. The bound is what the rates had with T from the species'
    enthalpies and ln A in the exponent (2.88e-15 and 4.18e-15 on these states)."""
    from pelelm_gb300.reactor import reaction_rates
    torch = cuda
    cfg = CONFIGS[cfgname]
    m, n = load_mechanism(cfg.mech), 4096
    cs = make_cells(cfg, n, seed=40)
    ld = np.longdouble
    R, R_cal = ld(R_ERG), ld(1.98720425864083)
    rY, rE, T = (cs.rY * 1e3).astype(ld), (cs.rE * 0.1).astype(ld), cs.T.astype(ld)
    lo, hi = (np.array([getattr(s, q) for s in m.species]).astype(ld) for q in ("low", "high"))
    W, Tmid = (np.array([getattr(s, q) for s in m.species]).astype(ld) for q in ("W", "Tmid"))
    rho = rY.sum(1)
    Y, h = rY / rho[:, None], rE / rho * ld(10) ** 4

    def thermo(T):
        t = T[:, None]
        a = np.where((t < Tmid)[:, :, None], lo[None], hi[None])
        hk = a[..., 0] + t * (a[..., 1] / 2 + t * (a[..., 2] / 3 + t * (a[..., 3] / 4 + t * a[..., 4] / 5))) + a[..., 5] / t
        ck = a[..., 0] + t * (a[..., 1] + t * (a[..., 2] + t * (a[..., 3] + t * a[..., 4])))
        sk = a[..., 0] * np.log(t) + t * (a[..., 1] + t * (a[..., 2] / 2 + t * (a[..., 3] / 3 + t * a[..., 4] / 4))) + a[..., 6]
        return hk, ck, hk - sk

    for _ in range(12):
        hk, ck, _ = thermo(T)
        T = T + np.clip((h - (Y * hk * (R * T)[:, None] / W).sum(1)) / (Y * ck * R / W).sum(1), -100, 100)
    g = thermo(T)[2]
    C = rho[:, None] / 1000 * Y / W
    wdot, total = np.zeros_like(C), C.sum(1)
    for r in m.reactions:
        def k(a):
            return ld(a.A) * T ** ld(a.beta) * np.exp(-ld(a.Ea) / (R_cal * T))
        kf, M = k(r.rate), total
        for s, eff in r.efficiencies.items():
            M = M + (ld(eff) - 1) * C[:, m.index(s)]
        if r.kind == "falloff":
            Pr, F = k(r.low) * M / kf, ld(1)
            if r.troe:
                a, T3, T1 = (ld(v) for v in r.troe[:3])
                Fc = (1 - a) * np.exp(-T / T3) + a * np.exp(-T / T1)
                if len(r.troe) > 3:
                    Fc = Fc + np.exp(-ld(r.troe[3]) / T)
                lF = np.log10(Fc)
                lP = np.log10(np.maximum(Pr, ld(1e-300))) - ld("0.4") - ld("0.67") * lF
                F = ld(10) ** (lF / (1 + (lP / (ld("0.75") - ld("1.27") * lF - ld("0.14") * lP)) ** 2))
            kf = kf * Pr / (1 + Pr) * F
        q, back = kf.copy(), kf * np.exp(np.minimum(
            sum(nu * g[:, m.index(s)] for s, nu in r.products.items()) - sum(nu * g[:, m.index(s)] for s, nu in r.reactants.items())
            - (sum(r.products.values()) - sum(r.reactants.values())) * np.log(ld(1.01325e6) / (R * T)), 700))
        for s, nu in r.reactants.items():
            q = q * C[:, m.index(s)] ** nu
        for s, nu in r.products.items():
            back = back * C[:, m.index(s)] ** nu
        q = (q - back if r.reversible else q) * (M if r.kind == "three_body" else ld(1))
        for side, sign in ((r.reactants, -1), (r.products, 1)):
            for s, nu in side.items():
                wdot[:, m.index(s)] += sign * nu * q
    ref = (wdot * W * 1000).T

    def t3(v, nc):
        return torch.tensor(np.ascontiguousarray(np.asarray(v).reshape(n, nc).T.reshape(nc, 1, 1, n)), device="cuda")

    out = torch.zeros(m.ns, 1, 1, n, dtype=torch.float64, device="cuda")
    reaction_rates(cfg.mech, ((0, 0, 0), (n - 1, 0, 0)), t3(cs.rY * 1e3, m.ns), t3(cs.rE * 0.1, 1), t3(cs.T, 1), None, out)
    got = out.cpu().numpy().reshape(m.ns, n).astype(ld)
    assert float(np.sqrt(((got - ref) ** 2).sum() / (ref ** 2).sum())) <= bound
