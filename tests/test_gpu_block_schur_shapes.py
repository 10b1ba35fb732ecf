"""The damped block-Schur solve at the edges of its tiles and segments: reduced dimensions around
multiples of the factor's 32 x 32 tiles, primary blocks of one to sixteen columns, eliminated blocks
without, with few and with many couplings, against the dense solve in numpy FP64.

The equations are well conditioned (priors of the size of the blocks): the CG's relative residual of
1e-12 is a relative error of at most 1e-10 in the steps, and an FP64 factor needs at most three
iterations to reach it."""
import numpy as np
import pytest

from plabundle_gb300.device import Gb300Context
from plabundle_gb300.schur import BlockNormalEquations, SchurComplementSolverOptions, solve_damped_schur_complement

pytestmark = pytest.mark.gpu


def _equations(P, pb, E, views, seed):
    rng = np.random.default_rng(seed)
    eq = BlockNormalEquations(P, E, pb, 3)
    for b in range(P):
        eq.addPrimaryResidualBlock(b, np.eye(pb) * (2.0 + rng.random()) * np.sqrt(max(1, E * min(views, P) / P)),
                                   rng.normal(size=pb) * 0.1)
    for e in range(E):
        k = 0 if e % 11 == 5 else min(P, views if e % 3 else 1)
        prim = np.sort(rng.choice(P, k, replace=False))
        for b in prim:
            eq.addResidualBlocks([int(b)], [rng.normal(size=(2, pb)) * 0.4], e, rng.normal(size=(2, 3)),
                                 rng.normal(size=2) * 0.1, rng.uniform(0.5, 1.5))
        eq.addEliminatedResidualBlock(e, np.eye(3) * 1.5, rng.normal(size=3) * 0.1)
    return eq


def _dense(eq, damping):
    d = eq.export()
    s = eq.sizes()
    P, pb, E = s["primaryBlockCount"], s["primaryBlockSize"], s["eliminatedBlockCount"]
    H, b = d["H"].copy(), -d["g"].copy()
    dg = np.diag(H).copy()
    np.fill_diagonal(H, np.where(dg != 0, dg * (1 + damping), 1.0))
    W = np.zeros((E, P * pb, 3))
    for (e, p), w in zip(d["coupling_index"], d["W"]):
        W[e, p * pb:(p + 1) * pb] += w
    V = d["Hee"].copy()
    for i in range(3):
        V[:, i, i] *= 1 + damping
    Vi = np.linalg.inv(V)
    for e in range(E):
        Y = W[e] @ Vi[e]
        H -= Y @ W[e].T
        b += Y @ d["ge"][e]
    x = np.linalg.solve(H, b)
    y = np.einsum("ekl,el->ek", Vi, -d["ge"] - np.einsum("eak,a->ek", W, x))
    return x, y.reshape(-1)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("P,pb,E,views", [(1, 1, 1, 1), (31, 1, 40, 4), (32, 1, 7, 32), (33, 1, 300, 3), (8, 8, 64, 8),
                                          (13, 5, 33, 2), (6, 16, 129, 6), (97, 1, 1000, 5), (20, 13, 400, 20),
                                          (50, 6, 2000, 3)])
def test_block_schur_over_shapes(P, pb, E, views, mixed):
    eq = _equations(P, pb, E, views, 17 * P + pb)
    x_ref, y_ref = _dense(eq, 1e-3)
    ctx = Gb300Context(0)
    x, y, rep = solve_damped_schur_complement(ctx, eq, 1e-3, SchurComplementSolverOptions(useMixedPrecision=mixed))
    assert rep["converged"] == 1
    if not mixed:
        assert rep["iterations"] <= 3
    assert np.linalg.norm(x - x_ref) <= 1e-10 * np.linalg.norm(x_ref)
    assert np.linalg.norm(y - y_ref) <= 1e-10 * np.linalg.norm(y_ref)
    ctx.close()


@pytest.mark.parametrize("at", [0, 2, 3, 6, 14, 30, 32, 37, 46])
def test_a_pivot_of_exactly_zero_is_shifted(at):
    """Columns `at` and `at + 1` are equal and their scaled entries are exactly one, so that the second
    pivot is exactly zero wherever it falls in a panel or tile: the factor is repeated with a small shift
    and the solve reaches the consistent system's residual (1e-12 of the right-hand side, three entries of
    rounding per row)."""
    pb, P = 16, 3
    eq = BlockNormalEquations(P, 1, pb, 3)
    H, g = np.zeros((P * pb, P * pb)), np.zeros(P * pb)
    rng = np.random.default_rng(at)
    for b in range(P):
        J = 2.0 * np.eye(pb)
        c = at - b * pb
        if 0 <= c < pb:
            J[:, c + 1] = J[:, c]
        r = rng.normal(size=pb)
        eq.addPrimaryResidualBlock(b, J, r)
        H[b * pb:(b + 1) * pb, b * pb:(b + 1) * pb] = J.T @ J
        g[b * pb:(b + 1) * pb] = J.T @ r
    eq.addEliminatedResidualBlock(0, np.eye(3), np.zeros(3))
    ctx = Gb300Context(0)
    x, _, _ = solve_damped_schur_complement(ctx, eq, 0.0, SchurComplementSolverOptions(useMixedPrecision=False))
    assert np.linalg.norm(H @ x + g) <= 1e-11 * np.linalg.norm(g)
