"""A mechanism that is not built in: launches of every size answer as the oracle does."""
import numpy as np
import pytest

import extra_mechs
from helpers import boxes_from_cells, gather, outliers_within_global_error, tol_ratio
from pelelm_gb300.reactor import ReactorBase, rhoh_to_temp
from pelelm_gb300.workloads import CONFIGS, load_mechanism, make_cells


REDUCED = {"mid_syn": extra_mechs.reduced("drm19_syn", "mid_syn", 14), "wide_syn": extra_mechs.reduced("gri_syn", "wide_syn", 33)}


@pytest.fixture(scope="session")
def extra(native_lib, tmp_path_factory):
    """(library, folder) of the extra mechanisms."""
    d = str(tmp_path_factory.mktemp("extra"))
    return extra_mechs.build(d, [extra_mechs.trio(), extra_mechs.jump(), *REDUCED.values()]), d


def _advance(torch, cfg, cs, shape, mech, options, small=None):
    boxes = boxes_from_cells(torch, cs, [shape])
    r = ReactorBase.create("ReactorCvode", mech, f"ode.rtol={cfg.rtol} ode.atol={cfg.atol} {options}")
    r.init(2, 1)
    r.react_boxes(boxes, cfg.dt, 0.0)
    torch.cuda.synchronize()
    nfail = r.stats()["nfail"]
    if small is not None:  # a small launch, or cells handed over
        route = r.last_route()
        assert route[0] if small else route[1] > 0
    r.close()
    return gather(boxes, cs.rY.shape[1]), nfail


# a small launch, and one whose last cells the small-launch kernel finishes; coefficients of 3
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(8, 8, 8), (23, 21, 19)])
@pytest.mark.parametrize("options", ["", "gb.mapping=thread"])
def test_coefficients_of_three_match_the_oracle(extra, oracle_mod, cuda, shape, options):
    so, d = extra
    cfg = CONFIGS["lidryer_amr120"]
    n = int(np.prod(shape))
    cs = make_cells(cfg, n, seed=3)
    with extra_mechs.library(so):
        (rYg, Tg, rEg, FCg), nfail = _advance(cuda, cfg, cs, shape, "trio_syn", f"gb.precision=fp64 {options}")
    om = oracle_mod.OracleMech(f"{d}/trio_syn.mech")
    rYo, To, rEo, FCo, nf = om.react(cs.rY, cs.rYsrc, cs.T, cs.rE, cs.rEsrc, cs.mask, cfg.dt, cfg.rtol, cfg.atol)
    assert nfail == 0 and nf == 0
    # the bounds of the built-in mechanisms' oracle tests
    within = (np.abs(Tg - To) <= 1e-6 * To) & (tol_ratio(rYg, rYo, cfg.rtol, cfg.atol).max(1) <= 1.0)
    assert within.mean() >= 0.999
    out = np.nonzero(~within)[0]
    outliers_within_global_error(om, cs, out, (rYg[out], Tg[out]), (rYo[out], To[out]), cfg.dt, cfg.rtol)


# one warp; two cells a warp; just above the small-launch limit, where the last cells of each warp change
# kernels; the roundings of both kernels are written out, so no compiler choice can tell them apart
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(5, 1, 1), (13, 9, 7), (17, 13, 11), (23, 21, 19)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_kernels_agree_bit_for_bit(extra, cuda, shape, precision):
    cfg = CONFIGS["lidryer_amr120"]
    cs = make_cells(cfg, int(np.prod(shape)), seed=8)
    with extra_mechs.library(extra[0]):
        a, fa = _advance(cuda, cfg, cs, shape, "trio_syn", f"gb.precision={precision}")
        b, fb = _advance(cuda, cfg, cs, shape, "trio_syn", f"gb.precision={precision} gb.mapping=thread")
    assert fa == fb == 0
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


# the same of a group of lanes (14 species) and a warp (33) a cell: a small launch and one that hands cells over
@pytest.mark.gpu
@pytest.mark.parametrize("mech,cfgname,mapping,shapes", [("mid_syn", "drm19_2M", "group", [(13, 9, 7), (23, 21, 19)]),
                                                        ("wide_syn", "gri_1M", "warp", [(13, 9, 2), (13, 9, 7)])])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_larger_mechanisms_agree_bit_for_bit(extra, cuda, mech, cfgname, mapping, shapes, precision):
    cfg = CONFIGS[cfgname]
    for shape, small in zip(shapes, (True, False)):
        cs = extra_mechs.reduced_cells(make_cells(cfg, int(np.prod(shape)), seed=8), load_mechanism(cfg.mech), REDUCED[mech])
        opts = f"gb.precision={precision} ode.max_steps=2000"
        with extra_mechs.library(extra[0]):
            a, fa = _advance(cuda, cfg, cs, shape, mech, opts, small)
            b, fb = _advance(cuda, cfg, cs, shape, mech, opts + f" gb.mapping={mapping}", None)
        assert fa == fb
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)


# enthalpies that jump at Tmid: targets between the two branches have a root on either side (a 5 K overlap),
# and the guess decides, as in the oracle's iteration from that guess
@pytest.mark.gpu
def test_the_guess_decides_where_enthalpy_jumps(extra, oracle_mod, cuda):
    torch = cuda
    so, d = extra
    om = oracle_mod.OracleMech(f"{d}/jump_syn.mech")
    rng = np.random.default_rng(2)
    n, ns = 256, 3
    Y = rng.uniform(0.1, 1.0, (n, ns))
    Y /= Y.sum(1, keepdims=True)
    T = np.where(np.arange(n) % 2 == 0, rng.uniform(1000.2, 1004.0, n), rng.uniform(996.0, 999.8, n))
    guess = T + np.where(T > 1000.0, 0.5, -0.5)
    h = np.array([om.mixture_h(t, y) for t, y in zip(T, Y)])
    rho = rng.uniform(0.2, 2.0, n)

    def t3(a, nc):
        return torch.tensor(np.ascontiguousarray(np.asarray(a).reshape(n, nc).T.reshape(nc, 1, 1, n)), device="cuda")

    Tg = t3(guess, 1)
    with extra_mechs.library(so):
        rhoh_to_temp("jump_syn", ((0, 0, 0), (n - 1, 0, 0)), t3(Y * rho[:, None], ns), t3(rho * h * 1e-4, 1), Tg)
        torch.cuda.synchronize()
    To = om.hy2t(h, Y, guess)
    np.testing.assert_allclose(To, T, rtol=1e-9)  # both sides have cells whose root is the guess's
    np.testing.assert_allclose(Tg.cpu().numpy().reshape(n), To, rtol=1e-9)
