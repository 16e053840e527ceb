"""The per-function calls on grids with boundary cells of every kind, against the kernel-form oracle
bit for bit: gauge, stage and structure cells carry a boundary entry where an outlet cell carries its
ordinal, and the routing call must tell them apart whether or not there are control structures.  Small
grids run one row a thread of the routing kernel, the larger ones two."""
from dataclasses import replace

import numpy as np
import pytest

from hydropol2d_b200 import synthetic as S
from tests.cases import random_terrain
from tests.test_gpu_parity import FIELDS, assert_same_state, make_pair
from tests.test_inflow import stage_case

pytestmark = pytest.mark.gpu

# (rows, columns) with one and with two rows a thread of the routing kernel
SIZES = [("fp32", (33, 61)), ("fp64", (33, 61)), ("fp32", (449, 461)), ("fp64", (1013, 1001))]


def _wet(case):
    """Water everywhere, so that outlets and boundary cells all flow from the first step."""
    rng = np.random.default_rng(3)
    return replace(case, d0=rng.uniform(20.0, 120.0, case.shape))


def _case(kind, shape):
    if kind == "inflow":
        return _wet(S.inflow_case(*shape))
    if kind == "stage":
        return _wet(stage_case(*shape))
    if kind == "inflow and stage":
        case = stage_case(*shape)
        flood = S.inflow_case(*shape).inflow
        keep = flood["gauge"] == 1   # the block on the plane, away from the stage cells
        case.inflow = dict(t_start=flood["t_start"], rates=flood["rates"][:, :1], rows=flood["rows"][keep],
                           cols=flood["cols"][keep], gauge=np.zeros(keep.sum(), np.int32))
        return _wet(case)
    return _wet(S.structures_case(*shape))


def _sequence(m, t, ts, k):
    """One pass of the reference's main loop over its separate functions; the new clock."""
    m.hydrology_step(ts)
    m.li_step(ts)
    new, vmax = m.cfl_dt()
    m.track_maxima(t + ts)
    m.set_clock(t + new, new, k + 1)
    return t + new, new, k + 1, vmax


def _follow(case, precision, steps):
    g, o = make_pair(case, precision)
    d = g.diag()
    clock = d["t"], d["time_step"], d["k"], 0.0
    for _ in range(steps):
        after = _sequence(g, *clock[:3])
        assert after == _sequence(o, *clock[:3])
        clock = after
        assert_same_state(g, o, FIELDS + ["hf3", "qo"])
    dg, do = g.diag(), o.diag()
    # sums in another order than the oracle's, in the state's precision per thread
    rel = 1e-5 if precision == "fp32" else 1e-9
    for v in ("rain_volume", "outlet_volume", "inflow_volume", "structure_volume"):
        assert dg[v] == pytest.approx(do[v], rel=rel, abs=1e-9), v
    assert dg["outlet_volume"] > 0
    g.close()


@pytest.mark.parametrize("precision,shape", SIZES)
@pytest.mark.parametrize("kind", ["inflow", "stage", "inflow and stage", "structures"])
def test_boundary_cells_of_the_routing_call(kind, precision, shape, hp2d_lib, oracle_lib):
    _follow(_case(kind, shape), precision, 6 if shape[0] < 100 else 3)


@pytest.mark.parametrize("precision,shape", SIZES[2:])
@pytest.mark.parametrize("scheme,critical", [(1, 0), (2, 1), (3, 0)])
def test_two_rows_a_thread_of_the_routing_call(scheme, critical, precision, shape, hp2d_lib, oracle_lib):
    case = random_terrain(*shape, seed=scheme, walls=True)
    case.params.update(flag_numerical_scheme=scheme, flag_critical=critical)
    _follow(case, precision, 2)
