"""Small launches (the kernel with more lanes per cell that reactor.cu chooses below its limit) give
the bits of the mechanism's large-launch mapping: states, energies and RHS counts of every cell."""
import numpy as np
import pytest

from pelelm_gb300.reactor import BoxArrays, ReactorBase
from pelelm_gb300.workloads import CONFIGS, make_cells


def _advance(torch, cfg, shape, options, deck, seed, masked):
    nx, ny, nz = shape
    n = nx * ny * nz
    cs = make_cells(cfg, n, seed=seed)
    ns = cs.rY.shape[1]

    def t(a, nc):
        return torch.tensor(np.ascontiguousarray(np.asarray(a).reshape(n, nc).T.reshape(nc, nz, ny, nx)), device="cuda")

    mask = None
    if masked:
        mask = torch.tensor(np.where(np.arange(n) % 7 == 3, -1, 1).astype(np.int32).reshape(1, nz, ny, nx), device="cuda")
    b = BoxArrays(((0, 0, 0), (nx - 1, ny - 1, nz - 1)), t(cs.rY, ns), t(cs.rYsrc, ns), t(cs.T, 1), t(cs.rE, 1),
                  t(cs.rEsrc, 1), t(np.zeros(n), 1), mask)
    if deck:
        options += " ode.atol=1e-5 peleLM.use_typ_vals_chem=1 cvode.max_order=4"
    r = ReactorBase.create("ReactorCvode", cfg.mech, options)
    r.init(2, 1)
    if deck:
        r.set_typ_vals_ode([max(1e-10, float(v)) for v in np.ptp(cs.rY, axis=0)] + [float(np.ptp(cs.T)) + 1.0])
    nfail = r.react(b.box, b.rY, b.rY_src, b.T, b.rEner, b.rEner_src, b.FC, mask, cfg.dt, 0.0)
    r.close()
    return nfail, b


# one cell; fewer cells than SMs; one cell a warp on every SM; two cells a warp (16-lane groups) and a
# remainder that leaves half a warp idle; just below the limit of the 9-species mechanism
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (13, 3, 2), (13, 9, 7), (17, 13, 11)])
@pytest.mark.parametrize("cfgname,mapping", [("lidryer_amr120", "thread"), ("drm19_2M", "group")])
@pytest.mark.parametrize("precision,deck,masked", [("mixed", False, False), ("fp64", False, True), ("mixed", True, True)])
def test_small_launch_bits(native_lib, cuda, shape, cfgname, mapping, precision, deck, masked):
    torch = cuda
    cfg = CONFIGS[cfgname]
    opts = f"gb.precision={precision}"
    fa, a = _advance(torch, cfg, shape, opts, deck, 5, masked)
    fb, b = _advance(torch, cfg, shape, opts + f" gb.mapping={mapping}", deck, 5, masked)
    assert fa == fb == 0
    assert torch.equal(a.FC, b.FC)
    assert torch.equal(a.rY, b.rY) and torch.equal(a.rEner, b.rEner) and torch.equal(a.T, b.T)


# above the small-launch limit: the last cells of each warp change to the small-launch kernel at a step
@pytest.mark.gpu
@pytest.mark.parametrize("cfgname,mapping", [("lidryer_amr120", "thread"), ("drm19_2M", "group")])
@pytest.mark.parametrize("precision,deck", [("mixed", False), ("fp64", True)])
def test_handed_over_cells_keep_their_bits(native_lib, cuda, cfgname, mapping, precision, deck):
    torch = cuda
    cfg = CONFIGS[cfgname]
    opts = f"gb.precision={precision}"
    fa, a = _advance(torch, cfg, (23, 21, 19), opts, deck, 9, True)
    fb, b = _advance(torch, cfg, (23, 21, 19), opts + f" gb.mapping={mapping}", deck, 9, True)
    assert fa == fb == 0
    for x, y in ((a.FC, b.FC), (a.rY, b.rY), (a.rEner, b.rEner), (a.T, b.T)):
        assert torch.equal(x, y)


# as many cells as lanes hold at once, the last warps part full: those would hand cells over before their
# first step, when the pivots are not yet set (they keep them until a step is done)
@pytest.mark.gpu
@pytest.mark.parametrize("cfgname,mapping", [("lidryer_amr120", "thread"), ("drm19_2M", "group")])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("shape", [(25, 17, 18), (29, 27, 22)])
def test_part_full_warps_keep_their_bits(native_lib, cuda, cfgname, mapping, precision, shape):
    torch = cuda
    cfg = CONFIGS[cfgname]
    assert 0 < np.prod(shape) % 32 <= 13
    opts = f"gb.precision={precision}"
    fa, a = _advance(torch, cfg, shape, opts, False, 4, False)
    fb, b = _advance(torch, cfg, shape, opts + f" gb.mapping={mapping}", False, 4, False)
    assert fa == fb == 0
    for x, y in ((a.FC, b.FC), (a.rY, b.rY), (a.rEner, b.rEner), (a.T, b.T)):
        assert torch.equal(x, y)


# teams of warps: one cell; fewer cells than SMs; two teams a block; above the limit, where the last
# cells of the launch change to teams at a step; steps limited, so that cells fail and are retried
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (7, 5, 4), (11, 5, 5), (11, 9, 5)])
@pytest.mark.parametrize("precision,steps", [("mixed", 2000), ("fp64", 2000), ("mixed", 90)])
def test_teams_of_warps_keep_the_bits(native_lib, cuda, shape, precision, steps):
    torch = cuda
    cfg = CONFIGS["gri_1M"]
    opts = f"gb.precision={precision} ode.max_steps={steps}"
    fa, a = _advance(torch, cfg, shape, opts, False, 3, True)
    fb, b = _advance(torch, cfg, shape, opts + " gb.mapping=warp", False, 3, True)
    assert fa == fb
    for x, y in ((a.FC, b.FC), (a.rY, b.rY), (a.rEner, b.rEner), (a.T, b.T)):
        assert torch.equal(x, y)
