"""The strip step where its two cells a lane, its records for cells outside the grid and its branches
for whole rows can go wrong, against the kernel-form oracle bit for bit: widths around a strip's 28
and 60 output columns, a row or two of cells, and depths below the smallest normal number in the step
whose clamp is off (tiles too)."""
from dataclasses import replace

import numpy as np
import pytest

from tests.cases import random_terrain
from tests.test_gpu_parity import FIELDS, assert_same_clock, assert_same_state, make_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("layout", [1, 2])
@pytest.mark.parametrize("shape", [(2, 3), (5, 28), (18, 29), (17, 59), (16, 60), (33, 61), (7, 119), (6, 121), (5, 122)])
def test_widths_around_a_strip(shape, layout, precision):
    g, o = make_pair(random_terrain(*shape, seed=sum(shape), walls=shape[0] > 6), precision)
    g.set_layout(layout)
    g.set_tuning(16)
    for chunk in (1, 2, 31):
        g.fused_steps(chunk)
        o.fused_steps(chunk)
        assert_same_state(g, o, FIELDS, f"{shape} after {chunk}")
        assert_same_clock(g, o)
    g.close()


@pytest.mark.parametrize("layout", [0, 1, 2])
def test_depths_below_the_smallest_normal_number(layout):
    ny, nx = 20, 70
    rng = np.random.default_rng(4)
    case = random_terrain(ny, nx, seed=9, rain=0.0)
    z = np.where(rng.random((ny, nx)) < 0.5, 0.0, case.z)      # level neighbours: face depths as small as the cells'
    d0 = 10.0 ** rng.uniform(-40, -33, (ny, nx))               # mm: 1e-43 .. 1e-36 m
    d0[rng.random((ny, nx)) < 0.2] = 50.0
    d0[0, nx - 1] = -1e-5                                      # an outlet cell below zero: no clamp in the first step
    case = replace(case, z=z, d0=d0)
    g, o = make_pair(case, "fp32")
    if layout:
        g.set_layout(layout)
        g.set_tuning(16)
    for chunk in (1, 1, 20):
        g.fused_steps(chunk)
        o.fused_steps(chunk)
        assert_same_state(g, o, FIELDS, f"layout {layout} after {chunk}")
        assert_same_clock(g, o)
    g.close()
