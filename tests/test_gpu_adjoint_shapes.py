"""The backward pass (pb_gpu_backward) for other numbers of intrinsic columns (0 to 9) and calibration groups
(0 to 4) than the workload of test_gpu_adjoint.py, with held tracks and cameras, tracks that are not
processed, and losses of the points and intrinsics, against the CPU implicit differentiation at the same
state, in FP64 and in mixed precision.

Both sides solve the exact Hessian H of the same state in FP64, so that a gradient's relative error is of
the order of the relative residual times the condition of the Jacobi-scaled H, which the test computes:
1e-13, at which the conjugate gradients stop, and 200 roundings (2^-53) for the sums over hundreds of rows.
1e-9 covers the rounding of the residuals and Jacobians that H is made of."""
import numpy as np
import pytest

import oracle as O
import orc_adjoint as A
from plabundle_gb300 import synth
from plabundle_gb300.adjoint import camera_centre_loss, newton_polish
from plabundle_gb300.device import Gb300Context
from plabundle_gb300.problem import ImageRobustLoss, SolveOptions

pytestmark = pytest.mark.gpu

# calibration groups, refined parameters, held tracks, held cameras, loss
CASES = [(0, "", 0, [], ImageRobustLoss.Huber), (0, "", 7, [3, 8], ImageRobustLoss.Cauchy),
         (1, "f", 0, [], ImageRobustLoss.Cauchy), (2, "fcr", 5, [2], ImageRobustLoss.Cauchy),
         (3, "fr", 0, [6], ImageRobustLoss.Huber), (4, "facrm", 9, [], ImageRobustLoss.Cauchy),
         (2, "c", 3, [], ImageRobustLoss.LeastSquares)]


def _options(refine, loss, mixed):
    o = SolveOptions()
    o.solver.imageRobustLoss = loss
    o.solver.imageRobustLossScalePixels = 1.5
    o.solver.maxIterations = 100
    o.backend.enablePlaMatrixMixedPrecision = mixed
    o.calibration.refineSharedFocalLength = "f" in refine
    o.calibration.refineSharedFocalAspectRatio = "a" in refine
    o.calibration.refineSharedPrincipalPoint = "c" in refine
    o.calibration.refineSharedRadialDistortion = "r" in refine
    o.calibration.refineSharedMetashapeParameters = "m" in refine
    return o


def _problem(groups, held_tracks, held_cameras):
    p = synth.aerial_grid_problem(seed=31 + groups, n_along=4, n_lines=4, n_points=240, n_groups=max(1, groups))
    if groups == 0:
        p.cameraCalibrationGroupIds = None
    rng = np.random.default_rng(groups)
    # held points and cameras where they belong
    p.fixedTrackIndices = sorted(int(t) for t in rng.choice(p.n_tracks, held_tracks, replace=False))
    p.points[p.fixedTrackIndices] = p.truth_points[p.fixedTrackIndices]
    p.fixedCameraIndices = list(held_cameras)
    p.cameras[held_cameras, :12] = p.truth_cameras[held_cameras, :12]
    # tracks that the gate of the initial error drops: their observations take no part
    for t in rng.choice(np.setdiff1d(np.arange(p.n_tracks), p.fixedTrackIndices), 4, replace=False):
        p.obs_u[p.track_offsets[t]:p.track_offsets[t + 1]] += 900.0 * rng.choice([-1, 1])
    return p


def _condition(H):
    d = np.sqrt(np.abs(H.diagonal()))
    e = np.linalg.eigvalsh((H / d[:, None]) / d[None, :])
    assert e[0] > 0
    return e[-1] / e[0]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("groups,refine,held_tracks,held_cameras,loss", CASES)
def test_backward_over_shapes(groups, refine, held_tracks, held_cameras, loss, mixed):
    p = _problem(groups, held_tracks, held_cameras)
    o = _options(refine, loss, mixed)
    ctx = Gb300Context(0)
    assert ctx.upload(p, o) == 0
    assert ctx.solve()["status"] in (1, 2)
    newton_polish(ctx, iterations=3)
    d = ctx.download()
    rng = np.random.default_rng(5)
    T = A.centre_targets(p.truth_cameras, 0.1, seed=4)
    _, gc = camera_centre_loss(d["cameras"], T)
    gp = rng.normal(size=(p.n_tracks, 3))
    ng = ctx.sizes()["intrinsic_blocks"]
    assert ng == (groups if refine else 0)
    cols = [q for q in range(9) if (int(ctx.copts.intrinsic_mask) >> q) & 1]
    gi = np.zeros((max(1, ng), 13))
    if ng:
        gi[:, cols] = rng.normal(size=(ng, len(cols))) * 1e-3
    out = ctx.backward(grad_cameras=gc, grad_points=gp, grad_intrinsics=gi if ng else None)

    orc = O.Oracle(p, o)
    adj = A.AdjointOracle(orc, d["cameras"], d["points"], d["intrinsics"] if ng else None)
    z = np.zeros(adj.n_vars)
    _, dL = adj.centre_loss(z, T)
    nc, nt = p.n_cameras, p.n_tracks
    r = np.linalg.norm(d["points"], axis=1) / 1000.0
    scale = r / np.arctan(r)
    kind = adj.kind[6 * nc:6 * nc + 3 * nt].reshape(nt, 3)
    # dL/dX in the chart of the track: free points move by s(X) per unit, held ones by one
    dL[6 * nc:6 * nc + 3 * nt] += (np.where(kind == 1, scale[:, None], 1.0) * np.where(kind > 0, gp, 0.0)).ravel()
    if ng:
        dL[adj.base_g:adj.base_g + 13 * ng] += gi.ravel()
    tot, _ = adj.implicit(dL, z)
    _, _, H = adj.system(z)
    tol = 1e-9 + (1e-13 + 200 * 2.0 ** -53) * _condition(H[adj.free][:, adj.free].toarray())
    assert tol < 1e-3

    def near(got, want):
        assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want), (np.linalg.norm(got - want) / np.linalg.norm(want), tol)

    near(out["observations"], adj.observation_gradient(tot, p.n_obs))
    near(out["initial_cameras"], adj.initial_pose_gradient(tot, p.cameras))
    gip = np.where(kind == 2, tot[6 * nc:6 * nc + 3 * nt].reshape(nt, 3), 0.0)
    if held_tracks:
        near(out["initial_points"], gip)
    else:
        assert not out["initial_points"].any()
    # observations that take no part, exactly zero, and again after a pass with another loss
    idle = (adj.kind[adj.base_o:adj.base_o + 2 * p.n_obs].reshape(-1, 2) == 0)
    assert idle.any() and not out["observations"][idle].any()
    again = ctx.backward(grad_cameras=2.0 * gc)
    assert not again["observations"][idle].any() and again["observations"].any()
    ctx.close()
