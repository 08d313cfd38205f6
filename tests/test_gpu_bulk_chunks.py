"""The bulk update walks rows in 16-byte chunks: rows whose last chunk is whole, partial
or their only one, uniform and per-voxel rates, alone and in a batch, against the
oracle (FP64 1e-12, FP32 1e-5 of each substrate's largest value)."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def problem(sides, S, mode, seed):
    rng = np.random.default_rng(seed)
    V = int(np.prod(sides))
    shape = S if mode == 1 else S * V
    return dict(name="bulk", dims=3, bbmin=(0, 0, 0), bbmax=tuple(20 * v for v in sides), voxel=(20, 20, 20), dt=0.05,
                D=rng.uniform(10, 1e4, S), decay=rng.uniform(0.01, 1.0, S), initial=np.zeros(S),
                field=rng.random((sides[2], sides[1], sides[0], S)), field_layout="interleaved", boundary=[],
                interior=None, bulk=(mode, rng.random(shape), rng.random(shape), 4 * rng.random(shape)), agents=None,
                compute_internalized=False)


def check(g, o, tol):
    fg, fo = g.get_field(), o.get_field()
    norm = np.abs(fo).reshape(-1, fo.shape[-1]).max(axis=0)
    assert (np.abs(fg - fo).reshape(-1, fo.shape[-1]) / norm).max() <= tol


@pytest.mark.parametrize("sides,S", [((1, 3, 2), 1), ((5, 3, 2), 1), ((3, 2, 5), 2), ((7, 4, 3), 3), ((4, 5, 3), 4),
                                     ((43, 3, 3), 3), ((130, 2, 2), 5)])
@pytest.mark.parametrize("mode", [1, 2])
def test_bulk_rows(pcg, oracle_mod, sides, S, mode):
    p = problem(sides, S, mode, S)
    o = W.apply(oracle_mod.OracleSolver(threads=2), p)
    o.solve(3)
    for prec, tol in ((pcg.FP64, 1e-12), (pcg.FP32, 1e-5)):
        alone, batched = W.apply(pcg.Solver(prec), p), W.apply(pcg.Solver(prec), p)
        alone.solve(3)
        pcg.Batch([batched]).solve(3)
        check(alone, o, tol)
        check(batched, o, tol)
