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
