"""Uniform bulk rates are applied in the last sweep's tiles where it has tiles enough, and
interior Dirichlet nodes then get their values' bulk update: solve() against the same
step in two calls (sweeps and faces, then the rest), which keeps the bulk pass apart
(the same bits), and against the oracle.  Meshes of at least 608 tiles of 32 columns
and of fewer, with conditions that hold for some substrates only."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides,S", [((70, 70, 9), 9), ((330, 61, 17), 2), ((1000, 9, 0), 20), ((20, 17, 12), 3)])
@pytest.mark.parametrize("prec", ["FP32", "FP64"])
def test_bulk_in_the_last_sweep(pcg, oracle_mod, sides, S, prec):
    rng = np.random.default_rng(S)
    dims = 3 if sides[2] else 2
    n = [max(v, 1) for v in sides]
    K = 60
    lin = rng.choice(n[0] * n[1] * n[2], K, replace=False)
    vox = np.stack([lin % n[0], (lin // n[0]) % n[1], lin // (n[0] * n[1])], axis=1)[:, :dims].astype(np.uint64)
    ag = W.agents_block(rng, 40, S, (vox[:40] + 0.5) * 20.0)  # agents on the nodes
    p = dict(name="bulk", dims=dims, bbmin=(0, 0, 0), bbmax=tuple(20 * v if a < dims else 0 for a, v in enumerate(n)),
             voxel=(20, 20, 20), dt=0.05, D=W.log_uniform(rng, 10, 1e4, S), decay=rng.uniform(0.01, 1.0, S),
             initial=np.zeros(S), field=rng.random((n[2], n[1], n[0], S)), field_layout="interleaved",
             boundary=[(0, 0, rng.random(S), np.ones(S, np.uint8)), (dims - 1, 1, rng.random(S), (rng.random(S) < 0.6))],
             interior=(vox, 3 * rng.random((K, S)), (rng.random((K, S)) < 0.7).astype(np.uint8)),
             bulk=(1, rng.random(S), rng.random(S), 4 * rng.random(S)), agents=ag, compute_internalized=True)
    g, h = (W.apply(pcg.Solver(getattr(pcg, prec)), p) for _ in range(2))
    o = W.apply(oracle_mod.OracleSolver(threads=2), p)
    o.solve(3)
    g.solve(3)
    for _ in range(3):
        h.run_phases(pcg.PHASE_DIFFUSION | pcg.PHASE_DIRICHLET, False)
        h.run_phases(pcg.PHASE_BULK | pcg.PHASE_CELLS, True)
    assert np.array_equal(g.get_field(), h.get_field())
    assert np.array_equal(g.get_internalized(), h.get_internalized())
    fo = o.get_field()
    norm = np.abs(fo).reshape(-1, S).max(axis=0)
    err = (np.abs(g.get_field() - fo).reshape(-1, S) / norm).max()
    assert err <= (1e-12 if prec == "FP64" else 1e-5)
