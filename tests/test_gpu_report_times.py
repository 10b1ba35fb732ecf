"""The phase times of the solve report (pb_solve_report): intervals of the solve's stream that follow one
another, so that each is positive where its work was done, zero where it was not, and their sum is at most
the time of the whole call, on every path: phases queued behind one another (a kept factor) or with waits
between them (a new factor for every iteration), online and general path, rigs, many trial steps, linear
solves that no step follows."""
import numpy as np
import pytest

from plabundle_gb300 import synth
from plabundle_gb300.device import Gb300Context
from plabundle_gb300.problem import ImageRobustLoss, SolveOptions

pytestmark = pytest.mark.gpu
PHASES = ("assembly_ms", "linear_ms", "back_substitution_ms", "objective_ms")


def _solve(p, reuse=0, mixed=True, linear_iterations=0, armijo=None):
    o = SolveOptions()
    o.solver.imageRobustLoss = ImageRobustLoss.Huber
    o.solver.imageRobustLossScalePixels = 1.5
    o.backend.enablePlaMatrixMixedPrecision = mixed
    o.backend.factorReuse = reuse
    o.backend.maxLinearIterations = linear_iterations
    if armijo is not None:
        o.solver.referenceArmijoCoefficient = armijo
    ctx = Gb300Context(0)
    assert ctx.upload(p, o) == 0
    ctx.solve()
    rep = ctx.solve()
    ctx.close()
    return rep


@pytest.mark.parametrize("reuse,mixed", [(0, True), (2, True), (1, False), (0, False)])
@pytest.mark.parametrize("layout", ["ring", "targets", "rig"])
def test_phases_follow_one_another(layout, reuse, mixed):
    if layout == "rig":
        p = synth.rig_grid_problem(seed=3, n_along=4, n_lines=2, n_points=1500)
    else:
        p = synth.ring_problem(seed=3, n_cameras=12, n_points=600)
        if layout == "targets":
            synth.with_control_points(p, n=6, sigma=0.02, seed=4)
    rep = _solve(p, reuse, mixed)
    assert rep["accepted_steps"] > 0
    t = np.array([rep[k] for k in PHASES])
    assert np.isfinite(t).all() and (t > 0).all()
    assert t.sum() <= rep["total_ms"]


@pytest.mark.parametrize("reuse", [0, 2])
def test_linear_solves_that_no_step_follows(reuse):
    # one CG iteration never reaches the tolerance: every iteration ends with its linear solve
    rep = _solve(synth.ring_problem(seed=3, n_cameras=12, n_points=600), reuse, True, linear_iterations=1)
    assert rep["accepted_steps"] == 0 and rep["rejected_steps"] == rep["iterations"] > 1
    assert rep["assembly_ms"] > 0 and rep["linear_ms"] > 0
    assert rep["back_substitution_ms"] == 0 and rep["objective_ms"] == 0
    assert rep["assembly_ms"] + rep["linear_ms"] <= rep["total_ms"]


def test_many_trial_steps():
    # an Armijo coefficient that no step length passes: every trial of the line search is evaluated
    rep = _solve(synth.ring_problem(seed=3, n_cameras=12, n_points=600), armijo=10.0)
    assert rep["accepted_steps"] == 0 and rep["objective_evaluations"] > 30
    assert 0 < rep["objective_ms"] < sum(rep[k] for k in PHASES) <= rep["total_ms"]
