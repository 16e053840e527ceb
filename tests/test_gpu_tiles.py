"""The tile form of the fused step (grids too small for strips) against the strip form, bit for bit:
sizes at the edges of the tiles (28 output columns, 12 / 19 / 8 output rows), one and two rows per
thread, both precisions, every kernel variant.  The strips themselves are held to the oracle by
test_gpu_layout.py; both run the same operations on the same values, so nothing may differ."""
import numpy as np
import pytest

from hydropol2d_b200 import synthetic as S
from tests.cases import random_terrain
from tests.conftest import same_bits
from tests.test_gpu_parity import FIELDS

pytestmark = pytest.mark.gpu

EXACT_DIAG = ["t", "time_step", "k", "max_velocity", "neg_depth_warnings", "unstable_steps", "rain_t0", "rain_t1",
              "t_previous", "status_bits"]


def _pair(case, precision):
    from hydropol2d_b200 import SurfaceFlow
    out = []
    for strips in (False, True):
        g = SurfaceFlow(*case.shape, case.resolution, precision, **case.params)
        case.apply(g)
        if strips:
            g.set_layout(2 if precision == "fp32" else 1)
            g.set_tuning(16)
        out.append(g)
    return out


def _same(a, b, extra=()):
    for f in list(FIELDS) + list(extra):
        assert same_bits(a.download_native(f), b.download_native(f)), f
    da, db = a.diag(), b.diag()
    for k in EXACT_DIAG:
        assert da[k] == db[k], k
    for k in ("rain_volume", "infiltration_volume", "outlet_volume", "inflow_volume", "structure_volume"):
        assert np.isclose(da[k], db[k], rtol=1e-6, atol=1e-9), k


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("shape", [(3, 4), (8, 27), (12, 28), (13, 29), (25, 57), (64, 85)])
def test_tile_edges(shape, precision, hp2d_lib):
    a, b = _pair(random_terrain(*shape, seed=sum(shape), walls=min(shape) > 8), precision)
    for chunk in (1, 3, 37):
        a.fused_steps(chunk)
        b.fused_steps(chunk)
        _same(a, b)


@pytest.mark.parametrize("precision,shape", [("fp32", (449, 461)), ("fp64", (1013, 1001))])
def test_two_rows_per_thread(precision, shape, hp2d_lib):
    a, b = _pair(random_terrain(*shape, seed=5, walls=True), precision)
    for chunk in (2, 35):
        a.fused_steps(chunk)
        b.fused_steps(chunk)
        _same(a, b)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("soil,maps", [(False, False), (True, False), (True, True)])
def test_boundary_cells_soil_and_maps(soil, maps, precision, hp2d_lib):
    case = S.structures_case(49, 61, minutes=20.0, soil=soil, maps=maps)
    a, b = _pair(case, precision)
    for g in (a, b):
        g.set_hazard_tracking(True)
    for chunk in (1, 34):
        a.fused_steps(chunk)
        b.fused_steps(chunk)
        _same(a, b, ["I", "T"] if soil else [])
        for f in ("vmax", "hazard_max"):
            assert same_bits(a.download(f), b.download(f)), f


@pytest.mark.parametrize("scheme,critical", [(2, 0), (3, 1)])
def test_diffusive_schemes_and_dry_tiles(scheme, critical, hp2d_lib):
    case = S.dambreak_case(70, 200, 5.0, seed=3, hours=0.2)
    case.params.update(flag_numerical_scheme=scheme, flag_critical=critical)
    a, b = _pair(case, "fp32")
    for chunk in (1, 2, 200):
        a.fused_steps(chunk)
        b.fused_steps(chunk)
        _same(a, b)
    assert a.diag()["skipped_read_cells"] > 0
