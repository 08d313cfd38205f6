"""FP64 lines are solved from both ends towards a meeting point, and the sweeps leave
their scale factors to the last one: line lengths around the split (one block, two
blocks, remainders), one- to three-dimensional meshes, more than 32 substrates, and
meshes whose factors every sweep applies itself, against the oracle."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def problem(sides, S, D, seed, dt=0.01):
    rng = np.random.default_rng(seed)
    dims = len(sides)
    n = list(sides) + [1] * (3 - dims)
    return dict(name="halves", dims=dims, bbmin=(0, 0, 0), bbmax=tuple(20 * v if a < dims else 0 for a, v in enumerate(n)),
                voxel=(20, 20, 20), dt=dt, D=D * rng.uniform(0.5, 1.5, S), decay=rng.uniform(0.01, 1.0, S),
                initial=np.zeros(S), field=rng.random((n[2], n[1], n[0], S)), field_layout="interleaved",
                boundary=[(dims - 1, 1, rng.random(S), np.ones(S, np.uint8))], interior=None, bulk=None, agents=None,
                compute_internalized=False)


def run(pcg, oracle_mod, p, steps=3):
    g = W.apply(pcg.Solver(pcg.FP64), p)
    g.set_mass_check(True)
    o = W.apply(oracle_mod.OracleSolver(threads=4), p)
    g.solve(steps)
    o.solve(steps)
    fg, fo = g.get_field(), o.get_field()
    norm = np.abs(fo).reshape(-1, fo.shape[-1]).max(axis=0)
    return float((np.abs(fg - fo).reshape(-1, fo.shape[-1]) / norm).max()), g.get_mass_check()["worst"].max()


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 23, 24, 25, 33, 72, 145])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_line_lengths(pcg, oracle_mod, n, axis):
    sides = [5, 6, 7]
    sides[axis] = n
    err, mass = run(pcg, oracle_mod, problem(sides, 3, 4e4, n))
    assert err <= 1e-12 and mass <= 1e-12


@pytest.mark.parametrize("sides,S", [((37,), 2), ((300,), 40), ((9, 41), 1), ((50, 18), 33), ((20, 19, 18), 35)])
def test_dims_and_substrates(pcg, oracle_mod, sides, S):
    err, mass = run(pcg, oracle_mod, problem(sides, S, 1e4, S))
    assert err <= 1e-12 and mass <= 1e-12


@pytest.mark.parametrize("sides,S", [((40,), 3), ((30, 25), 3), ((17, 26, 30), 2), ((12, 9, 11), 36)])
def test_factors_in_every_sweep(pcg, oracle_mod, sides, S):
    # r = dt D / h^2 up to about 3000: the product of two axes' factors is far below
    # 2^-20, so no factor is deferred.  Each side's relative error is bounded by
    # sweeps * eps * (1 + 4 r): 9 * 1.1e-16 * 1.2e4 = 1.2e-11
    err, _ = run(pcg, oracle_mod, problem(sides, S, 8e5, 3, dt=1.0))
    assert err <= 2.4e-11


def test_batch_of_both(pcg, oracle_mod):
    # deferred and undeferred domains, dimensions and more than 32 substrates together
    ps = [problem((17, 26, 30), 2, 1e4, 1), problem((40,), 3, 1e4, 2), problem((30, 25), 34, 1e4, 3),
          problem((12, 9, 11), 5, 8e5, 4, dt=1.0)]
    gs = [W.apply(pcg.Solver(pcg.FP64), p) for p in ps]
    pcg.Batch(gs).solve(3)
    for p, g in zip(ps, gs):
        o = W.apply(oracle_mod.OracleSolver(threads=4), p)
        o.solve(3)
        fo = o.get_field()
        norm = np.abs(fo).reshape(-1, fo.shape[-1]).max(axis=0)
        err = (np.abs(g.get_field() - fo).reshape(-1, fo.shape[-1]) / norm).max()
        assert err <= (2.4e-11 if p["dt"] == 1.0 else 1e-12)
