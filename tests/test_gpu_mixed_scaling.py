"""One FP64 sweep kernel serves the domains of a batch that apply their scale factors on an
axis and those that leave them to a later one: 1-D, 2-D and 3-D domains, short and long
lines, with deferred factors and without, alone and together give the same bits."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W

pytestmark = pytest.mark.gpu

DOMAINS = [((40,), 3, 8e5, 1.0), ((70,), 2, 1e3, 0.01), ((30, 25), 3, 8e5, 1.0), ((33, 90), 9, 1e5, 0.01),
           ((17, 26, 30), 2, 8e5, 1.0), ((24, 64, 65), 8, 1e5, 0.01), ((12, 9, 150), 5, 10.0, 0.01), ((9, 8, 7), 36, 1e4, 0.01)]


def problem(sides, S, D, dt, seed):
    rng = np.random.default_rng(seed)
    dims = len(sides)
    n = list(sides) + [1] * (3 - dims)
    return dict(name="mixed", dims=dims, bbmin=(0, 0, 0), bbmax=tuple(20 * v if a < dims else 0 for a, v in enumerate(n)),
                voxel=(20, 20, 20), dt=dt, D=D * rng.uniform(0.5, 1.5, S), decay=rng.uniform(0.01, 1.0, S),
                initial=np.zeros(S), field=rng.random((n[2], n[1], n[0], S)), field_layout="interleaved",
                boundary=[(dims - 1, 1, rng.random(S), np.ones(S, np.uint8))], interior=None, bulk=None, agents=None,
                compute_internalized=False)


@pytest.mark.parametrize("mass_check", [False, True])
@pytest.mark.parametrize("which", [range(8), [1, 3, 5, 6], [0, 2, 4], [5], [7, 5]])
def test_alone_and_together(pcg, which, mass_check):
    ps = [problem(*DOMAINS[d], d) for d in which]
    alone, batched = ([W.apply(pcg.Solver(pcg.FP64), p) for p in ps] for _ in range(2))
    for s in alone + batched:
        s.set_mass_check(mass_check)
    pcg.Batch(batched).solve(3)
    for a, b in zip(alone, batched):
        a.solve(3)
        assert np.array_equal(a.get_field(), b.get_field())
