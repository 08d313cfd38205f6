"""Which kernels apply uniform bulk rates: the last sweep where it has at least three tiles
of 32 columns per SM (no bulk launch of its own), the bulk kernel otherwise, for per-voxel
tables and when the call leaves a phase out."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def bulk_launches(pcg, sides, S, mode, prec, phases=None):
    rng = np.random.default_rng(S)
    dims = 3 if sides[2] else 2
    n = [max(v, 1) for v in sides]
    V = int(np.prod(n))
    k = S if mode == 1 else S * V
    p = dict(name="route", dims=dims, bbmin=(0, 0, 0), bbmax=tuple(20 * v if a < dims else 0 for a, v in enumerate(n)),
             voxel=(20, 20, 20), dt=0.05, D=np.full(S, 1e3), decay=np.full(S, 0.1), initial=np.ones(S), field=None,
             boundary=[], interior=None, bulk=(mode, rng.random(k), rng.random(k), rng.random(k)), agents=None,
             compute_internalized=False)
    s = W.apply(pcg.Solver(prec), p)
    s.set_kernel_timing(True)
    s.reset_kernel_stats()
    if phases is None:
        s.solve(2)
    else:
        s.run_phases(phases, False)
    s.synchronize()
    return s.kernel_stats()["bulk"]["launches"]


@pytest.mark.parametrize("prec", [0, 1])
def test_route(pcg, prec):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = -(-3 * sms // 2)  # two blocks of 32 columns a row
    assert bulk_launches(pcg, (8, rows, 9), 8, 1, prec) == 0
    assert bulk_launches(pcg, (8, rows - 1 if 2 * (rows - 1) < 3 * sms else rows - 2, 9), 8, 1, prec) == 2
    assert bulk_launches(pcg, (8, rows, 9), 8, 2, prec) == 2
    assert bulk_launches(pcg, (8 * 3 * sms, 5, 0), 4, 1, prec if 8 * 3 * sms * 4 * 8 < 200_000 else 0) == 0
    assert bulk_launches(pcg, (8, rows, 9), 8, 1, prec, pcg.PHASE_DIFFUSION | pcg.PHASE_BULK) == 1
