"""The objective kernels at the sizes where their launch shapes change (one cluster, one observation per
thread, several per thread) and at values at the edges of their bit-pattern tests, against the same
sum in plain numpy FP64.

A term's residual is a difference of pixel coordinates of a few thousand, so its square carries about
4 x 4000 x 2^-53 / |r| of relative error, at most 1e-11 for the residuals here; the terms are not
negative, so the sum carries no more."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-11


def _inputs(n, seed, extremes):
    rng = np.random.default_rng(seed)
    nc, npt = 7, max(1, n // 3)
    cams = np.zeros((nc, 32))
    for i in range(nc):
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        cams[i, 0:9] = (q * np.sign(np.linalg.det(q))).reshape(9)
    cams[:, 12:16] = (3500.0, 3400.0, 2000.0, 1500.0)
    cams[:, 16:21] = (-0.05, 0.01, -0.002, 1e-4, -2e-4)
    cams[:, 21:23] = 1.0
    cams[1, 21], cams[2, 22], cams[3, 23] = -1.0, -1.0, 1.0  # mirrored axes, forward along -z
    cam = rng.integers(0, nc, n)
    pt = np.sort(rng.integers(0, npt, n))
    # points in front of the camera of their first observation
    X = np.zeros((npt, 3))
    for i in range(npt):
        c = cam[np.searchsorted(pt, i)] if i in pt[:200] else int(rng.integers(0, nc))
        xc = np.array([rng.uniform(-1, 1), rng.uniform(-1, 1), rng.uniform(4, 9) * (-1 if cams[c, 23] else 1)])
        X[i] = cams[c, 0:9].reshape(3, 3) @ xc + cams[c, 9:12]
    u, v = rng.uniform(0, 4000, n), rng.uniform(0, 3000, n)
    w = rng.uniform(0.2, 3.0, n)
    if extremes:
        for k, val in enumerate((np.nan, np.inf, -1.0, 0.0, -0.0, 1e150, 1e-300)):
            w[k::97] = val
        u[11::101] = np.inf
    return cams, X, cam.astype(np.int32), pt.astype(np.int32), u, v, w


def _reference(cams, X, cam, pt, u, v, w, loss, scale):
    c = cams[cam]
    d = X[pt] - c[:, 9:12]
    with np.errstate(all="ignore"):
        xc = np.einsum("nij,ni->nj", c[:, 0:9].reshape(-1, 3, 3), d)
        z = xc[:, 2]
        front = np.where(c[:, 23] != 0, -z, z) > 1e-9
        x, y = xc[:, 0] / z, xc[:, 1] / z
        r2 = x * x + y * y
        rad = 1 + r2 * (c[:, 16] + r2 * (c[:, 17] + r2 * c[:, 18]))
        p1, p2 = c[:, 19], c[:, 20]
        px = np.where(c[:, 21] < 0, -1, 1) * c[:, 12] * (x * rad + 2 * p1 * x * y + p2 * (r2 + 2 * x * x)) + c[:, 14]
        py = np.where(c[:, 22] < 0, -1, 1) * c[:, 13] * (y * rad + p1 * (r2 + 2 * y * y) + 2 * p2 * x * y) + c[:, 15]
        s = w * ((px - u) ** 2 + (py - v) ** 2)
        c2 = scale * scale
        if loss == 0:
            rho = 0.5 * s
        elif loss == 1:
            rho = np.where(s <= c2, 0.5 * s, scale * np.sqrt(s) - 0.5 * c2)
        else:
            rho = 0.5 * c2 * np.log1p(s / c2)
        good = front & (s >= 0) & np.isfinite(s) & np.isfinite(rho)
    return rho[good].sum(), int((~good).sum())


@pytest.mark.parametrize("loss", [0, 1, 2])
@pytest.mark.parametrize("n,extremes,shift", [(1, False, 0), (33, False, 1), (2048, True, 0), (4096, False, 0),
                                              (4097, True, 1), (155_649, True, 0), (330_001, False, 1)])
def test_objective_over_its_launch_shapes(n, extremes, shift, loss):
    import torch
    from plabundle_gb300 import native
    L = native.load()
    cams, X, cam, pt, u, v, w = _inputs(n, 100 + n + loss, extremes)
    scale = 1.5
    ref, ref_bad = _reference(cams, X, cam, pt, u, v, w, loss, scale)
    # `shift`: the camera records start 8 bytes past a 16-byte boundary
    store = torch.zeros(cams.size + shift, dtype=torch.float64, device="cuda")
    store[shift:] = torch.from_numpy(cams.reshape(-1))
    dev = [torch.from_numpy(a).cuda() for a in (X, cam, pt, u, v, w)]
    cost, bad = C.c_double(-1.0), C.c_int64(-1)
    for _ in range(2):
        st = L.pb_gpu_objective_noalloc(store.data_ptr() + 8 * shift, cams.shape[0], dev[0].data_ptr(), X.shape[0],
                                        *(t.data_ptr() for t in dev[1:]), n, loss, scale,
                                        torch.cuda.current_stream().cuda_stream, C.byref(cost), C.byref(bad))
        assert st == 0
        assert bad.value == ref_bad
        np.testing.assert_allclose(cost.value, ref, rtol=RTOL)


@pytest.mark.parametrize("loss", [1, 2])
@pytest.mark.parametrize("scale", [1e-3, 1e100, 1e160, float("inf")])
def test_objective_over_extreme_loss_scales(loss, scale):
    """Scales whose square or its reciprocal leaves the range of FP64 take the plain loss."""
    import torch
    from plabundle_gb300 import native
    L = native.load()
    cams, X, cam, pt, u, v, w = _inputs(500, 9, False)
    ref, ref_bad = _reference(cams, X, cam, pt, u, v, w, loss, scale)
    dev = [torch.from_numpy(a).cuda() for a in (cams, X, cam, pt, u, v, w)]
    cost, bad = C.c_double(-1.0), C.c_int64(-1)
    st = L.pb_gpu_objective_noalloc(dev[0].data_ptr(), 7, dev[1].data_ptr(), X.shape[0],
                                    *(t.data_ptr() for t in dev[2:]), 500, loss, scale, None, C.byref(cost),
                                    C.byref(bad))
    assert st == 0 and bad.value == ref_bad
    np.testing.assert_allclose(cost.value, ref, rtol=RTOL)


@pytest.mark.parametrize("trials", [1, 2, 3, 8])
@pytest.mark.parametrize("points", [40, 6_000])
def test_trial_costs_over_batch_shapes(points, trials):
    """A batch of trial step lengths (a block row each) gives each trial the cost it has alone, to the
    rounding of sums split over another number of blocks."""
    from plabundle_gb300 import synth
    from plabundle_gb300.device import Gb300Context
    from plabundle_gb300.problem import ImageRobustLoss, Precision, SolveOptions
    p = synth.ring_problem(seed=3, n_cameras=9, n_points=points)
    o = SolveOptions()
    o.solver.imageRobustLoss = ImageRobustLoss.Cauchy
    o.solver.imageRobustLossScalePixels = 1.5
    ctx = Gb300Context(0)
    assert ctx.upload(p, o) == 0
    ctx.linearize_schur(1e-3, Precision.Fp64)
    ctx.solve_reduced()
    ctx.back_substitute()
    alphas = [0.75 ** k for k in range(trials)]
    batch = ctx.cost_batch(alphas)
    alone = np.array([ctx.cost_batch([a])[0] for a in alphas])
    np.testing.assert_allclose(batch, alone, rtol=1e-13)
    ctx.close()
