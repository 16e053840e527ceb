"""An ensemble whose row copies all time out (a wait limit of zero polls; every wait stays bounded and a
block that gives up waits for its copies): with more items than the GPU holds CTAs, the CTAs that gave
up leave items of the step untaken, and with fewer, the step's last item ends it.  Either way the call
reports HP2D_TIMEOUT, the step is not taken, and with the limit back the member goes on as if the
attempt had not been made, on its own and in the ensemble."""
import pytest

from tests.cases import random_terrain
from tests.conftest import same_bits
from tests.test_gpu_parity import FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(64, 256), (2600, 2600)])
def test_timed_out_ensemble_step_is_reported_and_not_taken(shape, hp2d_lib):
    from hydropol2d_b200 import HP2DError, SurfaceFlow
    from hydropol2d_b200.ensemble import Ensemble
    case = random_terrain(*shape, seed=8)
    ens = Ensemble()
    m, ref = (SurfaceFlow(*case.shape, case.resolution, "fp32", **case.params) for _ in range(2))
    for g in (m, ref):
        case.apply(g)
    ens.add(m)
    ens.steps(3)
    ref.fused_steps(3)
    m.set_wait_limit(0)
    for n in (1, 2, 40):   # a launch, launches, a graph
        with pytest.raises(HP2DError) as e:
            ens.steps(n)
        assert e.value.status_name == "HP2D_TIMEOUT"
        assert m.diag()["k"] == ref.diag()["k"]
    m.set_wait_limit(1 << 22)
    with pytest.raises(HP2DError) as e:   # the member's own call reports it once more and prepares the retry
        m.fused_steps(1)
    assert e.value.status_name == "HP2D_TIMEOUT"
    for f in FIELDS:
        assert same_bits(m.download_native(f), ref.download_native(f)), f
    ens.steps(3)
    m.fused_steps(2)
    ens.steps(2)
    ref.fused_steps(7)
    for f in FIELDS:
        assert same_bits(m.download_native(f), ref.download_native(f)), f
    dm, dr = m.diag(), ref.diag()
    for v in ("t", "time_step", "k", "max_velocity"):
        assert dm[v] == dr[v], v
    for v in ("rain_volume", "outlet_volume"):   # per-lane sums of other strips: FP32 with compensation
        assert dm[v] == pytest.approx(dr[v], rel=1e-5), v
    ens.close()
    ref.close()
