"""Ballots of a single domain: the sums of a shared voxel live in the row of its second
agent, counts are cleared over the voxels of the last ballot when agents are few, and
agents are listed 4 or 16 to a thread.  Crowds (whole warps in one voxel, pairs,
triples, everyone alone), one and many substrates, agent numbers around a thread's and
a block's share, and repeated ballots with moved and (de)activated agents, against the
oracle: counts bit-exact, fields and amounts within 1e-12 (FP64) and 1e-5 (FP32)."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SIDES = (24, 20, 18)


def positions(rng, A, crowd):
    ext = np.array(SIDES) * 20.0
    pos = W.uniform_positions(rng, A, 3, 0.0, ext)
    if crowd == "one":
        pos[:] = 20.0 * rng.integers(0, 18, 3) + rng.uniform(1, 19, (A, 3))
    elif crowd == "runs":  # agents in voxel order, 1 to 70 in a voxel
        v = np.repeat(np.arange(A), rng.integers(1, 71, A))[:A]
        pos = np.stack([v % 24, v // 24 % 20, v // 480 % 18], 1) * 20.0 + rng.uniform(1, 19, (A, 3))
    elif crowd == "triples":
        pos = pos[rng.integers(0, max(A // 3, 1), A)]
    return pos


@pytest.mark.parametrize("A", [1, 2, 3, 4, 5, 33, 1023, 1025, 4097])
@pytest.mark.parametrize("S,crowd", [(1, "none"), (3, "triples"), (4, "one"), (8, "runs"), (11, "triples"), (2, "runs")])
def test_repeated_ballots(pcg, oracle_mod, A, S, crowd):
    rng = np.random.default_rng(A * 100 + S)
    ag = W.agents_block(rng, A, S, positions(rng, A, crowd), secretion_hi=5.0, active_frac=0.9, net_export_hi=1.0)
    p = dict(name="ballot", dims=3, bbmin=(0, 0, 0), bbmax=tuple(20 * v for v in SIDES), voxel=(20, 20, 20), dt=0.01,
             D=W.log_uniform(rng, 10, 1e4, S), decay=rng.uniform(0.01, 1.0, S), initial=np.zeros(S),
             field=rng.random((SIDES[2], SIDES[1], SIDES[0], S)), field_layout="interleaved", boundary=[],
             interior=None, bulk=None, agents=ag, compute_internalized=True)
    o = W.apply(oracle_mod.OracleSolver(threads=2), p)
    gs = [(W.apply(pcg.Solver(pcg.FP64), p), 1e-12), (W.apply(pcg.Solver(pcg.FP32), p), 1e-5)]
    for turn in range(3):
        if turn:
            pos = positions(rng, A, crowd if turn == 1 else "none")
            act = (rng.random(A) < 0.8).astype(np.uint8)
            for s in [o] + [g for g, _ in gs]:
                s.update_agents(positions=pos, is_active=act)
                s.recompute_positional_data()
        o.solve(2)
        fo, io = o.get_field(), o.get_internalized()
        norm = np.abs(fo).reshape(-1, S).max(axis=0)
        for g, tol in gs:
            g.solve(2)
            assert np.array_equal(g.get_counts(), o.get_counts()) and g.get_conflict() == o.get_conflict()
            assert (np.abs(g.get_field() - fo).reshape(-1, S) / norm).max() <= tol
            den = np.abs(ag["uptake"] + ag["secretion"]).max() * 0.01 * 2494.0 / 8000.0 * max(1, o.get_counts().max())
            assert np.abs(g.get_internalized() - io).max() <= tol * 8000.0 * norm.max() * (1 + den)
