"""The tile step with two rows a thread against the strips, bit for bit: every kernel variant (gauge,
stage and structure cells, hazard maxima, soil, rain maps, the schemes with numerical diffusion, dry
tiles) and the largest grids of each kind that the size rule gives to the tiles.  The strips are held to
the oracle by test_gpu_layout.py and test_gpu_strip_edges.py."""
import numpy as np
import pytest

from hydropol2d_b200 import synthetic as S
from tests.cases import random_terrain
from tests.conftest import same_bits
from tests.test_gpu_tiles import _pair, _same
from tests.test_inflow import stage_case

pytestmark = pytest.mark.gpu

SIZES = [("fp32", (449, 461)), ("fp64", (1013, 1001))]   # just above one row a thread, off the tiles' sides


def _follow(case, precision, chunks, soil=False, hazard=False):
    pair = _pair(case, precision)
    if hazard:
        for g in pair:
            g.set_hazard_tracking(True)
    for chunk in chunks:
        for g in pair:
            g.fused_steps(chunk)
        _same(*pair, ["I", "T"] if soil else [])
        for f in ("vmax", "hazard_max") if hazard else ():
            assert same_bits(pair[0].download(f), pair[1].download(f)), f
    for g in pair:
        g.close()


@pytest.mark.parametrize("precision,shape", SIZES)
@pytest.mark.parametrize("soil,maps", [(False, False), (True, False), (False, True), (True, True)])
def test_structures_soil_and_maps(soil, maps, precision, shape, hp2d_lib):
    _follow(S.structures_case(*shape, soil=soil, maps=maps), precision, (1, 34), soil, hazard=True)


@pytest.mark.parametrize("precision,shape", SIZES)
def test_gauges_and_stages(precision, shape, hp2d_lib):
    case = stage_case(*shape)
    flood = S.inflow_case(*shape).inflow
    keep = flood["gauge"] == 1
    case.inflow = dict(t_start=flood["t_start"], rates=flood["rates"][:, :1] * 20.0, rows=flood["rows"][keep],
                       cols=flood["cols"][keep], gauge=np.zeros(keep.sum(), np.int32))
    case.d0 = np.random.default_rng(1).uniform(0.0, 60.0, shape)
    _follow(case, precision, (1, 34))


@pytest.mark.parametrize("precision,shape", SIZES)
@pytest.mark.parametrize("scheme,critical", [(2, 0), (3, 1)])
def test_schemes_with_diffusion(scheme, critical, precision, shape, hp2d_lib):
    case = random_terrain(*shape, seed=12, walls=True)
    case.params.update(flag_numerical_scheme=scheme, flag_critical=critical)
    _follow(case, precision, (2, 33))


@pytest.mark.parametrize("precision,shape", SIZES)
def test_dry_tiles(precision, shape, hp2d_lib):
    _follow(S.dambreak_case(*shape, 5.0, seed=3, hours=0.2), precision, (1, 2, 60))


@pytest.mark.parametrize("precision,shape,soil,maps", [("fp32", (1570, 1591), False, False), ("fp32", (1810, 1822), True, False),
                                                       ("fp32", (1810, 1822), False, True), ("fp32", (2610, 2603), True, True),
                                                       ("fp64", (2310, 2333), True, True)])
def test_largest_grids_on_tiles(precision, shape, soil, maps, hp2d_lib):
    _follow(S.structures_case(*shape, soil=soil, maps=maps), precision, (3,), soil)
