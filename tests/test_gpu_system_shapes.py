"""The reduced system, its dense copy and the point steps for other numbers of intrinsic columns (0 to 9),
calibration groups (1 to 4) and observations (ragged against warps and blocks) than the parity cases,
against the CPU FP64 oracle.

Tolerances: those of the parity tests.  FP64 entries 1e-9 of the diagonal scale (another order of
summation); mixed entries 2e-4 (FP32 Jacobians).  The oracle back-substitutes the step of the device, so
that the point steps differ by the elimination alone: FP64 1e-7 (rounding times the condition of a point
block, at most 1e6), mixed 2e-2 (FP32 rounding of the Jacobians times that of a damped point block)."""
import numpy as np
import pytest

import oracle as O
from plabundle_gb300 import synth
from plabundle_gb300.device import Gb300Context
from plabundle_gb300.problem import ImageRobustLoss, Precision, SolveOptions

pytestmark = pytest.mark.gpu

# calibration groups, refined parameters, points
CASES = [(0, "", 9), (0, "", 331), (1, "f", 60), (1, "fa", 251), (2, "c", 300), (3, "r", 400), (4, "fcr", 500),
         (2, "fcrm", 700), (1, "facrm", 333), (4, "facrm", 801)]


def _problem(groups, points):
    if groups == 0:
        return synth.ring_problem(seed=points, n_cameras=6, n_points=points)
    return synth.aerial_grid_problem(seed=points, n_along=4, n_lines=4, n_points=points, n_groups=groups)


def _options(refine, mixed):
    o = SolveOptions()
    o.solver.imageRobustLoss = ImageRobustLoss.Cauchy
    o.solver.imageRobustLossScalePixels = 1.5
    o.backend.enablePlaMatrixMixedPrecision = mixed
    o.calibration.refineSharedFocalLength = "f" in refine
    o.calibration.refineSharedFocalAspectRatio = "a" in refine
    o.calibration.refineSharedPrincipalPoint = "c" in refine
    o.calibration.refineSharedRadialDistortion = "r" in refine
    o.calibration.refineSharedMetashapeParameters = "m" in refine
    return o


@pytest.mark.parametrize("groups,refine,points", CASES)
@pytest.mark.parametrize("precision", [Precision.Fp64, Precision.Mixed])
def test_reduced_system_and_point_steps(groups, refine, points, precision):
    p = _problem(groups, points)
    o = _options(refine, precision == Precision.Mixed)
    ctx = Gb300Context(0)
    assert ctx.upload(p, o) == 0
    orc = O.Oracle(p, o, linear_solver=1)
    damping = 1e-2
    _, sg = ctx.linearize_schur(damping, precision)
    _, so = orc.build(damping)
    assert sg == so
    s = ctx.sizes()
    ncb, ng, ni = s["camera_blocks"], s["intrinsic_blocks"], s["ni"]
    cols = [q for q in range(9) if (int(ctx.copts.intrinsic_mask) >> q) & 1]
    assert len(cols) == ni and ng == (groups if refine else 0)
    m = np.array([13 * i + a for i in range(ncb) for a in range(6)] +
                 [13 * (ncb + g) + c for g in range(ng) for c in cols])
    S, rhs, direct = ctx.reduced()
    So, red = orc.dense_reduced()
    So = So[np.ix_(m, m)]
    d = np.sqrt(np.abs(np.diag(So)))
    d[d == 0] = 1.0
    tol = 1e-9 if precision == Precision.Fp64 else 2e-4
    assert np.abs((S - So) / np.outer(d, d)).max() < tol
    for got, want in ((rhs, -red["gradient"][m]), (direct, red["direct_rhs"][m])):
        assert np.abs((got - want) / d).max() < tol * max(1.0, np.abs(want / d).max())
    step, converged, _, _ = ctx.solve_reduced()
    assert converged
    padded = np.zeros(orc.info()["primary"] * 13)
    padded[m] = step
    elim, decrease, ok = ctx.back_substitute()
    oelim, odecrease, ook = orc.back_substitute(padded)
    assert ok and ook
    tol = 1e-7 if precision == Precision.Fp64 else 2e-2
    assert np.linalg.norm(elim - oelim) <= tol * np.linalg.norm(oelim)
    assert abs(decrease - odecrease) <= (1e-7 if precision == Precision.Fp64 else 1e-5) * abs(odecrease)


@pytest.mark.parametrize("n_along,n_lines", [(18, 18), (20, 17), (19, 18)])
def test_dense_copy_on_either_side_of_its_size_rule(n_along, n_lines):
    """1 954 unknowns are laid out on the device, 2 050 and 2 062 on the host.  The conjugate gradients stop at a
    relative residual of 2e-10 on the device's own matrix; the copy, multiplied here, adds the rounding of
    2 000 products a row."""
    p = synth.aerial_grid_problem(seed=n_along, n_along=n_along, n_lines=n_lines, n_points=6000, n_groups=2)
    ctx = Gb300Context(0)
    assert ctx.upload(p, _options("fcr", False)) == 0
    ctx.linearize_schur(1e-2, Precision.Fp64)
    S, rhs, _ = ctx.reduced()
    assert len(rhs) == 6 * (n_along * n_lines - 1) + 2 * ctx.sizes()["ni"] and np.array_equal(S, S.T)
    step, converged, _, _ = ctx.solve_reduced()
    assert converged
    assert np.linalg.norm(S @ step - rhs) <= 1e-9 * np.linalg.norm(rhs)
