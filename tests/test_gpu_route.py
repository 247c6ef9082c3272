"""Which kernel a call runs on: keys and the autotuner's pick fix it for every launch size."""
import numpy as np
import pytest

from helpers import boxes_from_cells, gather
from pelelm_gb300.reactor import ReactorBase
from pelelm_gb300.workloads import CONFIGS, make_cells


def _advance(torch, r, cfg, shape, seed):
    cs = make_cells(cfg, int(np.prod(shape)), seed=seed)
    boxes = boxes_from_cells(torch, cs, [shape])
    r.react_boxes(boxes, cfg.dt, 0.0)
    return gather(boxes, cs.rY.shape[1]), r.last_route()


def _reactor(cfg, options):
    r = ReactorBase.create("ReactorCvode", cfg.mech, f"ode.rtol={cfg.rtol} ode.atol={cfg.atol} {options}")
    r.init(2, 1)
    return r


# tuned on 64 cells, where a warp per cell is fastest, and on a box where the default is
@pytest.mark.gpu
@pytest.mark.parametrize("cfgname,default", [("lidryer_amr120", "thread"), ("drm19_2M", "group/8")])
@pytest.mark.parametrize("first", [(4, 4, 4), (32, 32, 16)])
def test_small_calls_keep_to_the_autotuners_pick(native_lib, cuda, cfgname, default, first):
    cfg = CONFIGS[cfgname]
    r = _reactor(cfg, "gb.autotune=1")
    _advance(cuda, r, cfg, first, 1)
    pick = r.tuning().split("-> ")[1].strip()
    a, route = _advance(cuda, r, cfg, (13, 9, 7), 2)
    assert route[0] == (pick == default)
    r.close()
    name, _, lanes = pick.partition("/")
    key = {"thread": "", "warp": f"gb.wpb={lanes}", "group": f"gb.group={lanes}"}[name]
    s = _reactor(cfg, f"gb.mapping={name} {key}")
    b, route = _advance(cuda, s, cfg, (13, 9, 7), 2)
    assert route == (False, 0)
    s.close()
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("key", ["gb.group=8", "gb.group=4", "gb.mapping=group", "gb.wpb=16", "gb.tpb=128"])
def test_layout_keys_fix_the_kernel(native_lib, cuda, key):
    cfg = CONFIGS["drm19_2M"]
    r = _reactor(cfg, key)
    assert _advance(cuda, r, cfg, (13, 9, 7), 3)[1] == (False, 0)
    r.close()


# cells per SM on either side of the lines, short and long advances, both precisions
@pytest.mark.gpu
@pytest.mark.parametrize("cfgname,precision,dt,below,above", [
    ("lidryer_amr120", "mixed", 1e-6, 40, 41), ("lidryer_amr120", "mixed", 1e-5, 48, 49),
    ("lidryer_amr120", "fp64", 1e-6, 28, 29), ("lidryer_amr120", "fp64", 1e-5, 48, 49),
    ("drm19_2M", "mixed", 1e-6, 34, 35), ("drm19_2M", "mixed", 1e-5, 40, 41), ("drm19_2M", "fp64", 1e-6, 40, 41),
    ("gri_1M", "mixed", 1e-6, 2, 3)])
def test_the_line_of_small_launches(native_lib, cuda, cfgname, precision, dt, below, above):
    cfg = CONFIGS[cfgname]
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    r = _reactor(cfg, f"gb.precision={precision} ode.max_steps=2000")
    for per_sm, small in ((below, True), (above, False)):
        n = sms * per_sm
        boxes = boxes_from_cells(cuda, make_cells(cfg, n, seed=6), [(n, 1, 1)])
        r.react_boxes(boxes, dt, 0.0)
        assert r.last_route()[0] == small
    r.close()
