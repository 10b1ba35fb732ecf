"""An iteration's solve, point steps and first objectives are queued behind its assembly while a kept factor
preconditions, and dropped where the assembly or the solve makes them void.  With kernel timing on
(pb_gpu_set_timing) the same driver waits after every phase instead and queues nothing ahead, so that either
way takes the same kernels on the same values: report, history and state are equal to the last bit.  More
launches with the queue than without show that something was queued and dropped."""
import numpy as np
import pytest

from plabundle_gb300 import synth
from plabundle_gb300.device import Gb300Context
from plabundle_gb300.problem import ImageRobustLoss, Precision, SolveOptions

pytestmark = pytest.mark.gpu


def _options(mixed=True, reuse=0, refine=False, online=True, iterations=30):
    o = SolveOptions()
    o.solver.imageRobustLoss = ImageRobustLoss.Huber
    o.solver.imageRobustLossScalePixels = 1.5
    o.solver.maxIterations = iterations
    o.solver.useReferenceOnlineSchur = online
    o.backend.enablePlaMatrixMixedPrecision = mixed
    o.backend.factorReuse = reuse
    o.calibration.refineSharedFocalLength = refine
    o.calibration.refineSharedPrincipalPoint = refine
    o.calibration.refineSharedRadialDistortion = refine
    return o


def _solve(p, o, timing):
    ctx = Gb300Context(0)
    assert ctx.upload(p, o) == 0
    ctx.set_timing(timing)
    rep = ctx.solve()
    out, hist = ctx.download(), ctx.history()
    ctx.close()
    return rep, out, hist


def _both(p, o):
    (ra, sa, ha), (rb, sb, hb) = _solve(p, o, False), _solve(p, o, True)
    for k in ra:
        if not k.endswith("_ms") and k != "gpu_kernel_launches":
            assert ra[k] == rb[k] or (ra[k] != ra[k] and rb[k] != rb[k]), (k, ra[k], rb[k])
    for k in ("iterations", "cost"):
        assert np.array_equal(ha[k], hb[k])
    for k in sa:
        assert np.array_equal(sa[k], sb[k], equal_nan=sa[k].dtype != bool), k
    return ra, ra["gpu_kernel_launches"] - rb["gpu_kernel_launches"]


def _aerial():
    return synth.aerial_grid_problem(seed=12, n_along=8, n_lines=5, n_points=4000)


@pytest.mark.parametrize("mixed,reuse", [(True, 0), (False, 1)])
@pytest.mark.parametrize("online", [True, False])
def test_nothing_dropped(mixed, reuse, online):
    rep, _ = _both(_aerial(), _options(mixed, reuse, True, online))
    assert rep["accepted_steps"] > 5


@pytest.mark.parametrize("mixed,reuse", [(True, 0), (False, 1)])
def test_rig_with_targets_and_bars(mixed, reuse):
    p = synth.rig_grid_problem(seed=7, n_along=5, n_lines=3, n_points=2500)
    synth.with_control_points(p, n=8, sigma=0.02, seed=8)
    synth.with_scale_bars(p, n=3, sigma=0.005, seed=9)
    rep, _ = _both(p, _options(mixed, reuse))
    assert rep["promoted_point_blocks"] > 0 and rep["accepted_steps"] > 3


@pytest.mark.parametrize("online", [True, False])
def test_kept_factor_that_does_not_converge(online):
    # a new factor needs at most about ten CG iterations here, a kept one about twenty
    o = _options(refine=True, online=online)
    o.backend.maxLinearIterations = 13
    rep, dropped = _both(_aerial(), o)
    assert rep["accepted_steps"] > 5 and dropped > 0


@pytest.mark.parametrize("online", [True, False])
def test_linear_solve_that_never_converges(online):
    o = _options(online=online, iterations=8)
    o.backend.maxLinearIterations = 1
    rep, dropped = _both(_aerial(), o)
    assert rep["accepted_steps"] == 0 and rep["rejected_steps"] == rep["iterations"] == 8 and dropped > 0


@pytest.mark.parametrize("online", [True, False])
def test_no_line_search_steps(online):
    o = _options(online=online, iterations=8)
    o.solver.referenceLineSearchSteps = 0
    rep, _ = _both(_aerial(), o)
    assert rep["accepted_steps"] == 0
    # the online path ends at the first step that is not accepted, the general path retries with more damping
    assert rep["iterations"] == (1 if online else 8)


@pytest.mark.parametrize("online", [True, False])
def test_line_search_beyond_the_queued_trial(online):
    o = _options(refine=True, online=online, iterations=6)
    o.solver.referenceArmijoCoefficient = 0.9  # (a decrease of nine tenths of the linear one: short steps)
    rep, _ = _both(_aerial(), o)
    assert rep["objective_evaluations"] > 3 * rep["iterations"]


def test_point_block_that_turns_singular():
    """A track of small weights, its point block's determinant at 0.9 of the 1e-15 that counts as singular:
    it passes with a damping of 0.1 and not with the next iteration's 0.01.  The solve starts a hundredth of a
    pixel from its solution, so that no step lowers the cost by the hundredth that discards a kept factor."""
    p = synth.ring_problem(seed=6, n_cameras=10, n_points=400, outlier_frac=0.0)
    o = _options(mixed=True, iterations=60)
    ctx = Gb300Context(0)
    assert ctx.upload(p, o) == 0
    ctx.solve()
    d = ctx.download()
    lin, at = ctx.linearize_observations(Precision.Fp64), ctx.active()
    ctx.close()
    t = int(np.nonzero((at["active_track"] == 1) & (at["track_block"] >= 0))[0][0])
    obs = slice(int(p.track_offsets[t]), int(p.track_offsets[t + 1]))
    J, w = lin["point_jacobian"][obs], lin["normal_weight"][obs]
    det = np.linalg.det(np.einsum("nri,n,nrj->ij", J, w, J))
    p.obs_weight[obs] *= (0.9e-15 / det) ** (1.0 / 3.0)
    rng = np.random.default_rng(2)
    p.cameras, p.points = d["cameras"].copy(), d["points"] + 3e-5 * rng.normal(size=p.points.shape)
    p.cameras[:, 9:12] += 3e-5 * rng.normal(size=(p.n_cameras, 3))
    rep, dropped = _both(p, o)
    assert rep["accepted_steps"] > 1 and rep["rejected_steps"] > 3 and dropped > 0
