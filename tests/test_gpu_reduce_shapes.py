"""The fixed-order sums of the chunk partials on either side of their dispatch: few lists (neighbours spread
over the blocks), many long lists (neighbours in one block), many short lists (a thread per entry), without
and with intrinsic columns, against the CPU FP64 oracle's reduced system.

Tolerances: those of the parity tests, entries within 1e-9 of the diagonal scale in FP64 (another order of
summation), 2e-4 in mixed precision (FP32 Jacobians)."""
import numpy as np
import pytest

import oracle as O
from plabundle_gb300 import synth
from plabundle_gb300.device import Gb300Context
from plabundle_gb300.problem import ImageRobustLoss, Precision, SolveOptions

pytestmark = pytest.mark.gpu

# layout, cameras (along, lines), points, refined
CASES = [("ring", (9, 1), 700, False), ("ring", (60, 1), 9000, False), ("ring", (75, 1), 24_000, False),
         ("aerial", (16, 10), 6000, False), ("aerial", (16, 10), 6000, True), ("aerial", (16, 10), 60_000, True)]


@pytest.mark.parametrize("layout,grid,points,refined", CASES)
@pytest.mark.parametrize("precision", [Precision.Fp64, Precision.Mixed])
def test_sums_of_the_partials(layout, grid, points, refined, precision):
    if layout == "ring":
        p = synth.ring_problem(seed=grid[0], n_cameras=grid[0], n_points=points, max_views=8, vectorized_views=True)
    else:
        p = synth.aerial_grid_problem(seed=points, n_along=grid[0], n_lines=grid[1], n_points=points, n_groups=2)
        if not refined:
            p.cameraCalibrationGroupIds = None
    o = SolveOptions()
    o.solver.imageRobustLoss = ImageRobustLoss.Huber
    o.solver.imageRobustLossScalePixels = 1.5
    o.backend.enablePlaMatrixMixedPrecision = precision == Precision.Mixed
    o.calibration.refineSharedFocalLength = o.calibration.refineSharedPrincipalPoint = refined
    o.calibration.refineSharedRadialDistortion = refined
    ctx = Gb300Context(0)
    assert ctx.upload(p, o) == 0
    ctx.linearize_schur(1e-2, precision)
    s = ctx.sizes()
    S, rhs, direct = ctx.reduced()
    ctx.linearize_schur(1e-2, precision)
    again = ctx.reduced()
    ctx.close()
    assert all(np.array_equal(a, b) for a, b in zip((S, rhs, direct), again))
    assert np.array_equal(S, S.T)
    orc = O.Oracle(p, o, linear_solver=1)
    orc.build(1e-2)
    ncb, ng = s["camera_blocks"], s["intrinsic_blocks"]
    cols = [q for q in range(9) if (int(ctx.copts.intrinsic_mask) >> q) & 1]
    m = np.array([13 * i + a for i in range(ncb) for a in range(6)] +
                 [13 * (ncb + g) + c for g in range(ng) for c in cols])
    assert len(m) == s["dim"] and ng == (2 if refined else 0)
    So, red = orc.dense_reduced()
    So = So[np.ix_(m, m)]
    d = np.sqrt(np.abs(np.diag(So)))
    d[d == 0] = 1.0
    tol = 1e-9 if precision == Precision.Fp64 else 2e-4
    assert np.abs((S - So) / np.outer(d, d)).max() < tol
    for got, want in ((rhs, -red["gradient"][m]), (direct, red["direct_rhs"][m])):
        assert np.abs((got - want) / d).max() < tol * max(1.0, np.abs(want / d).max())
