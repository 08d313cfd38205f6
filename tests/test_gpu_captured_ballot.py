"""A ballot that was only captured has not run: with few agents against voxels, the next
ballot must not clear the counts over voxels that no kernel has recorded, nor skip the
agents' terms.  The captured graph is replayed after it, agents moved in between;
counts are bit-exact with the oracle, fields within 1e-12 (FP64) and 1e-5 (FP32)."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SIDES = (24, 20, 18)


@pytest.mark.parametrize("prec,tol", [("FP32", 1e-5), ("FP64", 1e-12)])
@pytest.mark.parametrize("A", [1, 60, 530])  # fewer than one agent per 16 voxels
def test_captured_then_run(pcg, oracle_mod, A, prec, tol):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(A)
    S, ext = 3, np.array(SIDES) * 20.0
    pos = [W.uniform_positions(rng, A, 3, 0.0, ext) for _ in range(3)]
    pos[1][: A // 3] = pos[1][A // 3: 2 * (A // 3)]  # shared voxels
    p = dict(name="capture", dims=3, bbmin=(0, 0, 0), bbmax=tuple(20 * v for v in SIDES), voxel=(20, 20, 20), dt=0.01,
             D=np.array([1e3, 50.0, 2e4]), decay=np.array([0.1, 0.5, 1e-3]), initial=np.zeros(S),
             field=rng.random((SIDES[2], SIDES[1], SIDES[0], S)), field_layout="interleaved", boundary=[], interior=None,
             bulk=None, agents=W.agents_block(rng, A, S, pos[0], net_export_hi=1.0), compute_internalized=True)
    o = W.apply(oracle_mod.OracleSolver(threads=2), p)
    g = W.apply(pcg.Solver(getattr(pcg, prec)), p)
    stream = torch.cuda.Stream()
    g.set_stream(stream.cuda_stream)
    g.initialize()
    g.synchronize()

    def check():
        g.synchronize()
        fo = o.get_field()
        norm = np.abs(fo).reshape(-1, S).max(axis=0)
        assert np.array_equal(g.get_counts(), o.get_counts()) and g.get_conflict() == o.get_conflict()
        assert (np.abs(g.get_field() - fo).reshape(-1, S) / norm).max() <= tol

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        g.run_phases(pcg.PHASE_CELLS, True)
    for turn in range(3):  # the first ballots to run are not the captured one
        for s in (g, o):
            s.update_agents(positions=pos[turn])
            s.run_phases(pcg.PHASE_CELLS, True)
        check()
    for turn in (1, 2):
        for s in (g, o):
            s.update_agents(positions=pos[turn])
        o.run_phases(pcg.PHASE_CELLS, True)
        g.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        check()
        for s in (g, o):  # and a ballot of its own after the replay
            s.update_agents(positions=pos[turn - 1])
            s.run_phases(pcg.PHASE_CELLS, True)
        check()
