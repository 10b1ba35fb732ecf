"""A reduced system without unknowns (poses and intrinsics held) is refused by the dense solver: on the
first call of a context as on every later one, before and after the solve of another problem."""
import pytest

from plabundle_gb300 import synth
from plabundle_gb300.device import Gb300Context
from plabundle_gb300.problem import Precision, SolveOptions

pytestmark = pytest.mark.gpu


def _refused(ctx, p, mixed):
    o = SolveOptions()
    o.backend.enablePlaMatrixMixedPrecision = mixed
    o.calibration.refineCameraPose = False
    assert ctx.upload(p, o) == 0
    assert ctx.sizes()["dim"] == 0
    ctx.linearize_schur(1e-3, Precision.Mixed if mixed else Precision.Fp64)
    for _ in range(3):
        with pytest.raises(RuntimeError, match="dense factorisation failed"):
            ctx.solve_reduced()


@pytest.mark.parametrize("kind", ["ring", "rig"])
@pytest.mark.parametrize("mixed", [False, True])
def test_no_unknowns_is_refused_every_time(kind, mixed):
    if kind == "ring":
        p = synth.ring_problem(seed=3, n_cameras=7, n_points=60, max_views=4)
    else:
        p = synth.rig_grid_problem(seed=3, n_along=3, n_lines=2, n_points=200)
    ctx = Gb300Context(0)
    _refused(ctx, p, mixed)
    o = SolveOptions()
    o.backend.enablePlaMatrixMixedPrecision = mixed
    assert ctx.upload(p, o) == 0
    assert ctx.solve()["solution_usable"]
    _refused(ctx, p, mixed)
    ctx.close()
