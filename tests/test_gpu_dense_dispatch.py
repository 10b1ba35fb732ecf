"""Either side of the size rules of the dense factor and of the conjugate gradients, each solution checked
against the system it solves, in FP64 and mixed precision:

  factor      one cluster up to sixteen blocks (FP64 128 unknowns, FP32 320), a grid beyond; FP64 panels
              shared by four blocks up to 76 tiles (2 432 unknowns), one block a tile beyond
  CG          one cluster up to 384 unknowns with pose blocks, 320 without, a grid beyond

The reduced solve stops at a relative residual of 2e-10 on the device's matrix; the dense copy, multiplied
here, adds the rounding of up to 2 500 products a row.  The block-Schur solve stops at 1e-12; its equations
have a condition below 100, so that numpy's solution is within 1e-10."""
import numpy as np
import pytest

from plabundle_gb300 import synth
from plabundle_gb300.device import Gb300Context
from plabundle_gb300.problem import ImageRobustLoss, Precision, SolveOptions
from plabundle_gb300.schur import SchurComplementSolverOptions, solve_damped_schur_complement
from test_gpu_block_schur_shapes import _dense, _equations

pytestmark = pytest.mark.gpu


def _reduced(p, precision):
    o = SolveOptions()
    o.solver.imageRobustLoss = ImageRobustLoss.Cauchy
    o.solver.imageRobustLossScalePixels = 1.5
    o.backend.enablePlaMatrixMixedPrecision = precision == Precision.Mixed
    ctx = Gb300Context(0)
    assert ctx.upload(p, o) == 0
    ctx.linearize_schur(1e-2, precision)
    S, rhs, _ = ctx.reduced()
    step, converged, _, _ = ctx.solve_reduced()
    ctx.close()
    assert converged and np.array_equal(S, S.T)
    return len(rhs), np.linalg.norm(S @ step - rhs) / np.linalg.norm(rhs)


@pytest.mark.parametrize("precision", [Precision.Fp64, Precision.Mixed])
@pytest.mark.parametrize("cameras", [22, 23, 54, 55, 65, 66])
def test_pose_systems(cameras, precision):
    n, residual = _reduced(synth.ring_problem(seed=cameras, n_cameras=cameras, n_points=700), precision)
    assert n == 6 * (cameras - 1) and residual <= 1e-9


@pytest.mark.parametrize("n_along,n_lines", [(14, 29), (17, 24)])
def test_fp64_panels_shared_and_not(n_along, n_lines):
    p = synth.aerial_grid_problem(seed=n_lines, n_along=n_along, n_lines=n_lines, n_points=6000)
    p.cameraCalibrationGroupIds = None
    n, residual = _reduced(p, Precision.Fp64)
    assert n == 6 * (n_along * n_lines - 1) and residual <= 1e-9


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("P,pb", [(8, 16), (43, 3), (20, 16), (107, 3), (64, 6)])
def test_systems_without_pose_blocks(P, pb, mixed):
    eq = _equations(P, pb, 500, 4, P)
    x_ref, y_ref = _dense(eq, 1e-3)
    ctx = Gb300Context(0)
    x, y, rep = solve_damped_schur_complement(ctx, eq, 1e-3, SchurComplementSolverOptions(useMixedPrecision=mixed))
    ctx.close()
    assert rep["converged"] == 1
    assert np.linalg.norm(x - x_ref) <= 1e-10 * np.linalg.norm(x_ref)
    assert np.linalg.norm(y - y_ref) <= 1e-10 * np.linalg.norm(y_ref)
