"""Cells that change kernels at a step (the last ones of a large launch) end as they do in the launch's
own mapping, bit for bit: through failure and retry, I_R and graph replay. Each test sees to it that
cells were handed over."""
import numpy as np
import pytest

from helpers import boxes_from_cells, gather
from pelelm_gb300.reactor import ReactorBase
from pelelm_gb300.workloads import CONFIGS, make_cells

CASES = [("lidryer_amr120", "thread", (23, 21, 19)), ("drm19_2M", "group", (23, 21, 19)), ("gri_1M", "warp", (11, 11, 9))]


def _reactor(cfg, options):
    r = ReactorBase.create("ReactorCvode", cfg.mech, f"ode.rtol={cfg.rtol} ode.atol={cfg.atol} {options}")
    r.init(2, 1)
    return r


def _react(torch, cfg, shape, options):
    cs = make_cells(cfg, int(np.prod(shape)), seed=14)
    boxes = boxes_from_cells(torch, cs, [shape])
    r = _reactor(cfg, options)
    r.react_boxes(boxes, cfg.dt, 0.0)
    out = gather(boxes, cs.rY.shape[1]), r.stats(), r.last_route()
    r.close()
    return out


def _same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("cfgname,mapping,shape", CASES)
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_cells_are_handed_over(native_lib, cuda, cfgname, mapping, shape, precision):
    cfg = CONFIGS[cfgname]
    opts = f"gb.precision={precision} ode.max_steps=2000"
    a, sa, ra = _react(cuda, cfg, shape, opts)
    b, sb, rb = _react(cuda, cfg, shape, opts + f" gb.mapping={mapping}")
    assert not ra[0] and ra[1] > 0
    assert rb == (False, 0)
    assert sa == sb
    _same(a, b)


# the stiffest cells reach the step limit after they were handed over, and the FP64 pass takes them up
@pytest.mark.gpu
@pytest.mark.parametrize("cfgname,mapping,shape", CASES)
def test_handed_over_cells_that_fail(native_lib, cuda, cfgname, mapping, shape):
    cfg = CONFIGS[cfgname]
    _, s, _ = _react(cuda, cfg, shape, "")
    opts = f"ode.max_steps={int(0.8 * s['max_nst'])}"
    a, sa, ra = _react(cuda, cfg, shape, opts)
    b, sb, _ = _react(cuda, cfg, shape, opts + f" gb.mapping={mapping}")
    assert ra[1] > 0 and sa["nretry"] > 0
    assert sa == sb
    _same(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("cfgname,mapping,shape", CASES)
def test_i_r_of_handed_over_cells(native_lib, cuda, cfgname, mapping, shape):
    torch = cuda
    cfg = CONFIGS[cfgname]
    res = []
    for opts in ("", f"gb.mapping={mapping}"):
        cs = make_cells(cfg, int(np.prod(shape)), seed=15)
        cs.rY *= 1e3
        cs.rYsrc *= 1e3
        cs.rE *= 0.1
        cs.rEsrc *= 0.1
        boxes = boxes_from_cells(torch, cs, [shape])
        IR = torch.zeros_like(boxes[0].rY)
        r = _reactor(cfg, opts + " ode.max_steps=2000")
        r.advance_chemistry(boxes, cfg.dt, I_R=[IR])
        res.append((gather(boxes, cs.rY.shape[1]) + (IR.cpu().numpy(),), r.last_route()))
        r.close()
    assert res[0][1][1] > 0 and res[1][1][1] == 0
    _same(res[0][0], res[1][0])


# the counters start anew with each replay
@pytest.mark.gpu
@pytest.mark.parametrize("cfgname,mapping,shape", CASES)
def test_hand_over_in_graph_replays(native_lib, cuda, cfgname, mapping, shape):
    torch = cuda
    cfg = CONFIGS[cfgname]
    b, _, _ = _react(cuda, cfg, shape, f"ode.max_steps=2000 gb.mapping={mapping}")
    cs = make_cells(cfg, int(np.prod(shape)), seed=14)
    boxes = boxes_from_cells(torch, cs, [shape])
    fields = [boxes[0].rY, boxes[0].T, boxes[0].rEner]
    old = [f.clone() for f in fields]
    stream = torch.cuda.Stream()
    r = _reactor(cfg, "gb.graph=1 ode.max_steps=2000")
    for _ in range(3):
        for f, o in zip(fields, old):
            f.copy_(o)
        torch.cuda.synchronize()
        r.react_boxes(boxes, cfg.dt, 0.0, stream=stream)
        stream.synchronize()
        assert r.last_route()[1] > 0
        _same(gather(boxes, cs.rY.shape[1]), b)
    r.close()
