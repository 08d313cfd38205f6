"""pcg_estimate_device_bytes, which sizes a context's allocation and is what a server admits
by, against the buffers that a context has: the field and its transfer staging, a table
of three head rows per substrate and axis (FP64: and the scale factors), Dirichlet and bulk
tables, agents with their ballot scratch.  It covers them and exceeds them by the unused
part of the longest heads and a few KB only."""
import numpy as np
import pytest

from physicore_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def up(v, m):
    return (v + m - 1) // m * m


def buffers(sides, S, A, K, w):
    """Bytes of a context's buffers, coefficient heads at their longest."""
    dims = len(sides)
    n = list(sides) + [1] * (3 - dims)
    V, pitch = n[0] * n[1] * n[2], up(n[0] * S, 32 // w)
    parts = [n[1] * n[2] * pitch * w, V * S * w, 32, 32, max(S, 2) * 8, 6 * S * w, 6 * S]
    for a in range(dims):
        if w == 4:
            parts.append((3 * S * up(n[a], 8) + 7 * up(S, 4)) * w)
        else:
            m = n[a] if n[a] <= 8 else (n[a] + 8) // 16 * 8
            parts.append((3 * S * up(max(m, n[a] - m), 8) + 5 * S + n[a] * S) * w)
    parts += [8 * K, K * S * w, K * S]
    if A:
        ts = up(3 * S * w, 16)
        parts += [A * S * 8] * 6 + [A * dims * 8, A * 8, A, 4 * A, 4 * A, A, 4 * A, 4 * A, 12 * up(A, 4), A * ts, A * ts, 4 * V, 4 * V]
    return sum(parts)


@pytest.mark.parametrize("prec,w", [("FP32", 4), ("FP64", 8)])
@pytest.mark.parametrize("sides,S,A,K", [((8000,), 2, 0, 0), ((900, 3), 8, 0, 0), ((20, 19, 18), 3, 5000, 40), ((5, 6, 300), 20, 33, 0),
                                         ((9, 7, 5), 40, 1, 3), ((64, 60, 50), 1, 20000, 0)])
def test_estimate(pcg, sides, S, A, K, prec, w):
    rng = np.random.default_rng(S)
    dims = len(sides)
    s = pcg.Solver(getattr(pcg, prec))
    s.set_mesh(dims, (0, 0, 0), tuple(20 * v for v in sides) + (0,) * (3 - dims), (20,) * 3)
    s.set_substrates(0.01, np.full(S, 1e5), np.full(S, 0.1), np.zeros(S))
    if K:
        vox = np.stack([np.arange(K) % v for v in sides[:1]] + [np.arange(K) // sides[0] % v for v in sides[1:2]]
                       + [np.zeros(K, int)] * (dims - 2), axis=1)
        s.set_dirichlet_interior(vox.astype(np.uint64), np.ones((K, S)), np.ones((K, S), np.uint8))
    if A:
        ag = W.agents_block(rng, A, S, W.uniform_positions(rng, A, dims, 0.0, np.array(sides) * 20.0))
        s.set_agents(ag["positions"], ag["secretion"], ag["saturation"], ag["uptake"], ag["net_export"], ag["volumes"],
                     ag["is_active"])
    need, est = buffers(sides, S, A, K, w), s.estimate_device_bytes()
    assert need <= est <= need + 2048 + 16 * S * 3 * w * dims + 6 * S * (w + 1)
    s.solve(1)
    s.synchronize()
    s.close()
