"""A mechanism that is not built in: launches of every size answer as the oracle does."""
import numpy as np
import pytest

import extra_mechs
from helpers import boxes_from_cells, gather, outliers_within_global_error, tol_ratio
from pelelm_gb300.reactor import ReactorBase
from pelelm_gb300.workloads import CONFIGS, make_cells


@pytest.fixture(scope="session")
def extra(native_lib, tmp_path_factory):
    """(library, folder) of the extra mechanisms."""
    d = str(tmp_path_factory.mktemp("extra"))
    return extra_mechs.build(d, [extra_mechs.trio()]), d


def _advance(torch, cfg, cs, shape, mech, options):
    boxes = boxes_from_cells(torch, cs, [shape])
    r = ReactorBase.create("ReactorCvode", mech, f"ode.rtol={cfg.rtol} ode.atol={cfg.atol} {options}")
    r.init(2, 1)
    r.react_boxes(boxes, cfg.dt, 0.0)
    torch.cuda.synchronize()
    nfail = r.stats()["nfail"]
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
