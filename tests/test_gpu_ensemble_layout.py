"""A grid that was stepped in an ensemble (whose items are strips) keeps its own layout when it is
stepped alone again: the cells that the dry flags let its steps leave alone are counted by that layout's
units, tile by tile on a small grid, so they are those of a grid that was never in an ensemble."""
import pytest

from tests.cases import small_dambreak
from tests.conftest import same_bits
from tests.test_gpu_parity import FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuned", [False, True])
def test_member_keeps_its_own_layout(tuned, hp2d_lib):
    from hydropol2d_b200 import SurfaceFlow
    from hydropol2d_b200.ensemble import Ensemble
    case = small_dambreak(150, 400, seed=6)
    ens = Ensemble()
    m, ref = (SurfaceFlow(*case.shape, case.resolution, "fp32", **case.params) for _ in range(2))
    for g in (m, ref):
        case.apply(g)
        if tuned:
            g.set_layout(2)   # strips of its own
    ens.add(m)
    for _ in range(2):   # into the ensemble and back
        ens.steps(5)
        ref.fused_steps(5)
        counts = []
        for g in (m, ref):
            if tuned:
                g.set_tuning(32)
            g.fused_steps(6)   # the flags of the layout are set anew
            before = g.diag()
            g.fused_steps(40)
            after = g.diag()
            counts.append([after[v] - before[v] for v in ("skipped_cells", "skipped_read_cells")])
        assert counts[0] == counts[1]
        assert counts[0][1] > 0
        for f in FIELDS:
            assert same_bits(m.download_native(f), ref.download_native(f)), f
    ens.close()
    ref.close()
