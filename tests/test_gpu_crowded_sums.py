"""Sums of the agents of crowded voxels.  A voxel's agents are summed 32 at a time in pairs
(at most 5 roundings) and the k / 32 parts one after another, so the sum of k equal
terms is off by at most 5 + k / 64 units of roundoff u (the parts' running sum grows
evenly), and by u each for the terms' own rounding, for their FP64 evaluation and for
the last addition: (8 + k / 64) u.  Fields start at zero and nothing is taken up or
secreted, so the field of a voxel after one cell pass is the sum of its agents' exports.
A serial sum of 1,000 equal FP32 terms is off by 200 u."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W
from test_zz_no_alloc import Caller, _fn

pytestmark = pytest.mark.gpu

SIDES = (16, 14, 12)
COUNTS = [1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 24, 25, 31, 32, 33, 63, 64, 65, 127, 128, 129, 160, 161, 289, 1000, 5000]
ROUNDOFF = {"FP32": 2.0 ** -24, "FP64": 2.0 ** -53}


def crowds(rng, counts, order):
    """Positions of counts[c] agents in the c-th of random distinct voxels, shuffled or
    voxel by voxel, and those voxels."""
    lin = rng.choice(int(np.prod(SIDES)), len(counts), replace=False)
    v = np.stack([lin % SIDES[0], lin // SIDES[0] % SIDES[1], lin // (SIDES[0] * SIDES[1])], axis=1)
    who = np.repeat(np.arange(len(counts)), counts)
    if order == "shuffled":
        rng.shuffle(who)
    return (v[who] + rng.uniform(0.05, 0.95, (len(who), 3))) * 20.0, v


def problem(rng, pos, S, field=0.0, **rates):
    A = len(pos)
    ag = W.agents_block(rng, A, S, pos)
    for k in ("secretion", "uptake", "net_export"):  # every agent the same
        ag[k][:] = rates.get(k, np.zeros(S))
    return dict(name="crowd", dims=3, bbmin=(0, 0, 0), bbmax=tuple(20 * v for v in SIDES), voxel=(20, 20, 20), dt=0.01,
                D=np.full(S, 1e3), decay=np.full(S, 0.1), initial=np.zeros(S),
                field=np.full((SIDES[2], SIDES[1], SIDES[0], S), field), field_layout="interleaved", boundary=[],
                interior=None, bulk=None, agents=ag, compute_internalized=True)


def check(field, v, counts, net, u):
    got = field[v[:, 2], v[:, 1], v[:, 0]]
    k = np.array(counts, dtype=np.float64)[:, None]
    want = k * (net * 0.01 / 8000.0)
    err = np.abs(got - want) / want
    assert (err <= (8 + k / 64) * u).all(), (err / u).max(axis=1)


@pytest.mark.parametrize("prec", ["FP32", "FP64"])
@pytest.mark.parametrize("order", ["shuffled", "sorted"])
@pytest.mark.parametrize("S", [1, 2, 3, 4, 5, 8, 11, 20])
def test_sums_of_equal_terms(pcg, S, order, prec):
    rng = np.random.default_rng(S)
    pos, v = crowds(rng, COUNTS, order)
    net = rng.uniform(1.0, 2.0, S)
    s = W.apply(pcg.Solver(getattr(pcg, prec)), problem(rng, pos, S, net_export=net))
    s.run_phases(pcg.PHASE_CELLS, True)
    check(s.get_field(), v, COUNTS, net, ROUNDOFF[prec])
    assert s.get_counts().sum() == len(pos) and s.get_conflict()


@pytest.mark.parametrize("S", [3, 4])
def test_sums_in_caller_buffers(pcg, S):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(S)
    pos, v = crowds(rng, COUNTS, "shuffled")
    net = rng.uniform(1.0, 2.0, S)
    L, noalloc = _fn(pcg)
    caller = Caller(torch, problem(rng, pos, S, net_export=net), SIDES[0] * S)
    assert caller.call(noalloc) == 0, L.pcg_last_error().decode()
    torch.cuda.synchronize()
    check(caller.get_field(), v, COUNTS, net, ROUNDOFF["FP32"])


@pytest.mark.parametrize("prec", ["FP32", "FP64"])
def test_more_than_a_million_agents(pcg, prec):
    # eight agents to a thread, and a crowd of 100,000 among many small ones
    rng = np.random.default_rng(5)
    counts = [100_000] + list(rng.integers(1, 900, 2300))
    pos, v = crowds(rng, counts, "shuffled")
    assert len(pos) > 1 << 20
    net = rng.uniform(1.0, 2.0, 1)
    s = W.apply(pcg.Solver(getattr(pcg, prec)), problem(rng, pos, 1, net_export=net))
    s.run_phases(pcg.PHASE_CELLS, True)
    check(s.get_field(), v, counts, net, ROUNDOFF[prec])


@pytest.mark.parametrize("S", [1, 4, 11])
def test_crowds_against_the_oracle(pcg, oracle_mod, S):
    # 20,000 equal agents in four voxels: fields and amounts within 1e-5 in FP32
    rng = np.random.default_rng(S)
    pos, _ = crowds(rng, [5000] * 4, "shuffled")
    p = problem(rng, pos, S, field=0.5, secretion=rng.uniform(0.1, 1.0, S), uptake=rng.uniform(0.1, 0.5, S),
                net_export=rng.uniform(1.0, 50.0, S))
    g = W.apply(pcg.Solver(pcg.FP32), p)
    o = W.apply(oracle_mod.OracleSolver(threads=4), p)
    for s in (g, o):
        s.run_phases(pcg.PHASE_CELLS, True)
        s.run_phases(pcg.PHASE_CELLS, False)
    fo, io = o.get_field(), o.get_internalized()
    assert (np.abs(g.get_field() - fo) / np.abs(fo).reshape(-1, S).max(axis=0)).max() <= 1e-5
    assert (np.abs(g.get_internalized() - io).max(axis=0) <= 1e-5 * 8000.0 * np.abs(fo).reshape(-1, S).max(axis=0)).all()
