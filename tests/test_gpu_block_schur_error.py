"""The rounding of the FP64 block-Schur solve against the same equations in extended precision (`longdouble`:
113 bits on the GPU machine, 64 on x86), beside that of a plain FP64 evaluation that subtracts one eliminated
block's term after another.  The device adds the terms of a primary block in segments; both round every term
and every addition once, a segment's sum over fewer and smaller partial sums, so that the device's error is of
the size of the plain evaluation's.  Both are sums of thousands of independent roundings: a factor of two
covers the scatter of a mean over six sets of equations."""
import numpy as np
import pytest

from plabundle_gb300.device import Gb300Context
from plabundle_gb300.schur import BlockNormalEquations, SchurComplementSolverOptions, solve_damped_schur_complement

pytestmark = pytest.mark.gpu


def _equations(P, pb, E, views, seed):
    rng = np.random.default_rng(seed)
    eq = BlockNormalEquations(P, E, pb, 3)
    for b in range(P):
        eq.addPrimaryResidualBlock(b, np.eye(pb) * rng.uniform(0.5, 1.5), np.zeros(pb))
    for e in range(E):
        for b in np.sort(rng.choice(P, views, replace=False)):
            eq.addResidualBlocks([int(b)], [rng.normal(size=(2, pb)) * 0.5], e, rng.normal(size=(2, 3)),
                                 rng.normal(size=2) * 0.1, rng.uniform(0.5, 1.5))
    return eq


def _system(eq, damping, dtype):
    """The reduced system in `dtype`, one eliminated block's term after another."""
    d, s = eq.export(), eq.sizes()
    P, pb, E = s["primaryBlockCount"], s["primaryBlockSize"], s["eliminatedBlockCount"]
    H, b = d["H"].astype(dtype), -d["g"].astype(dtype)
    i = np.arange(P * pb)
    H[i, i] *= dtype(1) + dtype(damping)
    V = d["Hee"].astype(dtype)
    for k in range(3):
        V[:, k, k] *= dtype(1) + dtype(damping)
    rows, blocks = [[] for _ in range(E)], [[] for _ in range(E)]
    for (e, p), w in zip(d["coupling_index"], d["W"]):
        rows[e].append(np.arange(p * pb, (p + 1) * pb))
        blocks[e].append(w.astype(dtype))
    for e in range(E):
        r, W, v = np.concatenate(rows[e]), np.concatenate(blocks[e]), V[e]
        c = np.array([[v[1, 1] * v[2, 2] - v[1, 2] * v[2, 1], v[0, 2] * v[2, 1] - v[0, 1] * v[2, 2], v[0, 1] * v[1, 2] - v[0, 2] * v[1, 1]],
                      [v[1, 2] * v[2, 0] - v[1, 0] * v[2, 2], v[0, 0] * v[2, 2] - v[0, 2] * v[2, 0], v[0, 2] * v[1, 0] - v[0, 0] * v[1, 2]],
                      [v[1, 0] * v[2, 1] - v[1, 1] * v[2, 0], v[0, 1] * v[2, 0] - v[0, 0] * v[2, 1], v[0, 0] * v[1, 1] - v[0, 1] * v[1, 0]]])
        Y = W @ (c / (v[0] @ c[:, 0]))
        H[np.ix_(r, r)] -= Y @ W.T
        b[r] += Y @ d["ge"][e].astype(dtype)
    return H, b


def _refined(H, b):
    H64, x = H.astype(np.float64), np.zeros_like(b)
    for _ in range(6):
        x = x + np.linalg.solve(H64, (b - H @ x).astype(np.float64))
    return x


@pytest.mark.parametrize("P,pb,E,views", [(10, 13, 700, 5), (24, 13, 500, 4), (16, 7, 1200, 6)])
def test_split_sums_round_no_worse_than_a_plain_evaluation(P, pb, E, views):
    ctx = Gb300Context(0)
    device, plain = [], []
    for seed in range(6):
        eq = _equations(P, pb, E, views, seed)
        x, _, rep = solve_damped_schur_complement(ctx, eq, 1e-3, SchurComplementSolverOptions())
        assert rep["converged"] == 1
        want = _refined(*_system(eq, 1e-3, np.longdouble))
        H, b = _system(eq, 1e-3, np.float64)
        size = np.linalg.norm(want.astype(np.float64))
        device.append(np.linalg.norm((x - want).astype(np.float64)) / size)
        plain.append(np.linalg.norm((np.linalg.solve(H, b) - want).astype(np.float64)) / size)
    ctx.close()
    assert np.mean(device) <= 2 * np.mean(plain), (device, plain)
