"""Kernels of a step start as their predecessors leave, and the persistent sweeps clear
their own tile counters: the same steps with an event between any two kernels (which
keeps them apart) and replayed from a captured graph give the same bits.  No agents
share a voxel, so nothing is summed in any order."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def problem(sides, S, seed):
    rng = np.random.default_rng(seed)
    dims = len(sides)
    n = list(sides) + [1] * (3 - dims)
    V = int(np.prod(n))
    lin = rng.choice(V, min(V // 2, 200), replace=False)
    vox = np.stack([lin % n[0], (lin // n[0]) % n[1], lin // (n[0] * n[1])], axis=1)[:, :dims]
    half = len(lin) // 2
    ag = W.agents_block(rng, half, S, (vox[:half] + 0.5) * 20.0)
    return dict(name="chain", dims=dims, bbmin=(0, 0, 0), bbmax=tuple(20 * v if a < dims else 0 for a, v in enumerate(n)),
                voxel=(20, 20, 20), dt=0.01, D=W.log_uniform(rng, 10, 1e5, S), decay=rng.uniform(0.01, 1.0, S),
                initial=np.zeros(S), field=rng.random((n[2], n[1], n[0], S)), field_layout="interleaved",
                boundary=[(0, 0, rng.random(S), np.ones(S, np.uint8))],
                interior=(vox[half:].astype(np.uint64), rng.random((len(lin) - half, S)),
                          np.ones((len(lin) - half, S), np.uint8)),
                bulk=(1, rng.random(S), rng.random(S), rng.random(S)), agents=ag, compute_internalized=True)


# a few tiles, about one per resident CTA, and several per CTA
@pytest.mark.parametrize("sides,S", [((30,), 2), ((70, 40), 3), ((20, 19, 18), 1), ((96, 90, 64), 2), ((130, 120, 100), 4)])
@pytest.mark.parametrize("prec", ["FP32", "FP64"])
def test_chained_and_replayed_steps(pcg, sides, S, prec):
    torch = pytest.importorskip("torch")
    p = problem(sides, S, len(sides) * 10 + S)
    a, b, c = (W.apply(pcg.Solver(getattr(pcg, prec)), p) for _ in range(3))
    for s in (a, b, c):
        s.set_mass_check(True)
    a.solve(2)
    a.solve(6)
    b.set_kernel_timing(True)
    b.solve(8)
    stream = torch.cuda.Stream()
    c.synchronize()
    c.set_stream(stream.cuda_stream)
    c.solve(2)  # the ballot, and the first launches
    c.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        c.solve(2)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    want = b.get_field()
    assert np.array_equal(a.get_field(), want) and np.array_equal(c.get_field(), want)
    assert np.array_equal(a.get_internalized(), b.get_internalized())
    assert np.array_equal(c.get_internalized(), b.get_internalized())
