"""Chained kernels of ballots with shared voxels: the lists, flags and sums that one kernel
writes are read by the next ones.  Agents in pairs, in small crowds and alone are moved
between calls, alone and in a batch; counts and conflict flags are bit-exact with the
oracle, fields within 1e-12 (FP64) and 1e-5 (FP32) of each substrate's largest value."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SIDES = (30, 26, 22)


def positions(rng, A, crowd):
    pos = W.uniform_positions(rng, A, 3, 0.0, np.array(SIDES) * 20.0)
    return pos[rng.integers(0, max(A // crowd, 1), A)] if crowd > 1 else pos


@pytest.mark.parametrize("prec,tol", [("FP32", 1e-5), ("FP64", 1e-12)])
@pytest.mark.parametrize("A,S", [(200, 3), (700, 1), (900, 8), (5000, 4), (20000, 2)])
@pytest.mark.parametrize("batched", [False, True])
def test_moved_ballots(pcg, oracle_mod, A, S, prec, tol, batched):
    rng = np.random.default_rng(A + S)
    ag = W.agents_block(rng, A, S, positions(rng, A, 2), active_frac=0.9, net_export_hi=1.0)
    p = dict(name="chain", dims=3, bbmin=(0, 0, 0), bbmax=tuple(20 * v for v in SIDES), voxel=(20, 20, 20), dt=0.01,
             D=W.log_uniform(rng, 10, 1e4, S), decay=rng.uniform(0.01, 1.0, S), initial=np.zeros(S),
             field=rng.random((SIDES[2], SIDES[1], SIDES[0], S)), field_layout="interleaved", boundary=[],
             interior=None, bulk=None, agents=ag, compute_internalized=True)
    o = W.apply(oracle_mod.OracleSolver(threads=4), p)
    g = W.apply(pcg.Solver(getattr(pcg, prec)), p)
    step = pcg.Batch([g]) if batched else g
    for turn, crowd in enumerate([2, 5, 1, 30, 1, 2]):
        pos = positions(rng, A, crowd)
        for s in (g, o):
            s.update_agents(positions=pos)
            s.recompute_positional_data()
        step.solve(1)
        o.solve(1)
        fo = o.get_field()
        norm = np.abs(fo).reshape(-1, S).max(axis=0)
        assert np.array_equal(g.get_counts(), o.get_counts()) and g.get_conflict() == o.get_conflict(), turn
        assert (np.abs(g.get_field() - fo).reshape(-1, S) / norm).max() <= tol, turn
