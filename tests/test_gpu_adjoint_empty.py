"""The backward pass and the Newton step of a problem whose tracks all fail the gate of the initial error, so
that no observation takes part and the chunk plan is one empty chunk: the refined state does not depend on
the observations, the final camera poses are the initial ones, and only the priors hold the intrinsics."""
import numpy as np
import pytest

from plabundle_gb300 import synth
from plabundle_gb300.device import Gb300Context
from plabundle_gb300.problem import SolveOptions

pytestmark = pytest.mark.gpu


def _context(mixed, refined):
    p = synth.aerial_grid_problem(seed=4, n_along=4, n_lines=3, n_points=80, n_groups=2)
    p.obs_u = p.obs_u + 5000.0 * np.resize([1.0, -1.0], p.n_obs)
    o = SolveOptions()
    o.backend.enablePlaMatrixMixedPrecision = mixed
    o.calibration.refineSharedFocalLength = o.calibration.refineSharedPrincipalPoint = refined
    ctx = Gb300Context(0)
    assert ctx.upload(p, o) == 0
    s = ctx.sizes()
    assert s["observation_count"] == 0 and s["dim"] == (2 * s["ni"] if refined else 0) and s["camera_blocks"] == 0
    ctx.solve()
    return p, ctx


@pytest.mark.parametrize("mixed", [False, True])
def test_gradients_without_observations(mixed):
    p, ctx = _context(mixed, True)
    g = np.random.default_rng(1).normal(size=(p.n_cameras, 6))
    out = ctx.backward(grad_cameras=g)
    assert not out["observations"].any() and not out["initial_points"].any()
    assert np.array_equal(out["initial_cameras"], g)
    step, norm = ctx.newton_step()
    assert abs(step) <= 1e-9 and abs(norm) <= 1e-9  # (the priors are met by the initial values)
    ctx.close()


@pytest.mark.parametrize("mixed", [False, True])
def test_nothing_to_solve_is_refused(mixed):
    p, ctx = _context(mixed, False)
    with pytest.raises(RuntimeError):
        ctx.backward(grad_cameras=np.ones((p.n_cameras, 6)))
    with pytest.raises(RuntimeError):
        ctx.newton_step()
    assert ctx.download()["cameras"].shape == p.cameras.shape  # (the context is still usable)
    ctx.close()
