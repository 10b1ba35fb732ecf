"""The work that a user of this backend has it do, as measurable cases.

A case names a kind of work, a layout of the block and its sizes:

  objective   pb_gpu_objective_noalloc: the robust objective of caller-owned device arrays
  schur       one linearisation and point elimination, and the dense copy of the reduced system
              (normal equations for a covariance analysis or a caller's own solver)
  step        one Gauss-Newton / Levenberg-Marquardt step through the per-kernel entry points:
              linearise, eliminate, solve, back-substitute, evaluate the trial costs
  backward    the gradients of a loss of the refined camera centres with respect to every
              observation and initial pose, at a converged state
  solve       Solver.solve of a whole problem with a kept workspace
  rig         Solver.solve of an oblique rig block with control points and scale bars
  blockschur  the damped Schur solve of block normal equations that a caller assembled on the host

Layouts: "ring", cameras on a circle around a point cloud (Huber loss, known calibration), and
"aerial", a nadir flight grid (Cauchy loss, calibration groups with refined f, cx, cy, k1-k3, p1,
p2, or none).  Both follow the problems of plabundle_gb300.synth; the inputs are drawn on the GPU so
that a block of a million observations is ready in a fraction of a second.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from plabundle_gb300 import native, synth
from plabundle_gb300.adjoint import newton_polish
from plabundle_gb300.device import Gb300Context
from plabundle_gb300.problem import ImageRobustLoss, Precision, Problem, SolveOptions
from plabundle_gb300.schur import (BlockNormalEquations, SchurComplementSolverOptions,
                                   solve_damped_schur_complement)
from plabundle_gb300.solver import Solver, SolverWorkspace

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64


def listed():
    return [
        # a real-time loop's objective of a small local map: launch latency
        dict(name="objective_small", kind="objective", layout="ring", cameras=20, observations=2_001, points=450),
        # the same call at the largest input that it takes
        dict(name="objective_large", kind="objective", layout="aerial", cameras=500, observations=4_000_000,
             points=600_000),
        # normal equations of a close-range block in double precision
        dict(name="schur_ring_fp64", kind="schur", layout="ring", cameras=40, points=9_001, views=6, groups=0,
             mixed=False, damping=1e-3),
        # normal equations of a dense self-calibrating survey block, mixed precision
        dict(name="schur_aerial_mixed", kind="schur", layout="aerial", cameras=100, points=120_000, views=10,
             groups=2, mixed=True, damping=0.0),
        # one step of the smallest common problem, in double precision
        dict(name="step_ring_fp64", kind="step", layout="ring", cameras=20, points=2_000, views=6, groups=0,
             mixed=False, damping=0.0, trials=1),
        # one step of a mid-size block with a full batch of trial step lengths
        dict(name="step_aerial_mid", kind="step", layout="aerial", cameras=63, points=15_013, views=10, groups=1,
             mixed=True, damping=1e-2, trials=8),
        # one step of the self-calibrating 500-camera / 200 000-point aerial block
        dict(name="step_aerial_500", kind="step", layout="aerial", cameras=500, points=200_000, views=10, groups=2,
             mixed=True, damping=1e-3, trials=1),
        # gradients of a survey block's refined camera centres with respect to its measurements
        dict(name="backward_aerial", kind="backward", layout="aerial", cameras=60, points=20_000, views=10, groups=0,
             mixed=True),
        # a whole small solve with a kept workspace: upload, planning, iterations, download
        dict(name="solve_ring", kind="solve", layout="ring", cameras=20, points=2_000, views=6, groups=0, mixed=True),
        # a whole survey solve: five-camera rigs, control points, scale bars, general path
        dict(name="solve_rig", kind="rig", layout="rig", cameras=150, points=40_000, views=8, groups=0, mixed=True),
        # block normal equations of a caller that assembles on the host
        dict(name="blockschur", kind="blockschur", layout="host", blocks=40, eliminated=3_000, views=5, mixed=False,
             damping=1e-3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["objective", "schur", "step", "schur", "step", "backward", "solve", "blockschur"])
    if kind == "objective":
        layout = rng.choice(["ring", "aerial"])
        n = _log(rng, 500, 4_000_000)
        return dict(kind=kind, layout=layout, cameras=_log(rng, 8, 500), observations=n, points=max(50, n // 6))
    if kind == "blockschur":
        return dict(kind=kind, layout="host", blocks=_log(rng, 8, 60), eliminated=_log(rng, 200, 3_000),
                    views=rng.randint(3, 6), mixed=rng.random() < 0.5, damping=10.0 ** rng.randint(-4, -1))
    if kind == "solve":
        return dict(kind=kind, layout="ring", cameras=rng.randint(10, 60), points=_log(rng, 1_000, 20_000),
                    views=rng.randint(5, 8), groups=0, mixed=True)
    layout = "aerial" if kind == "backward" else rng.choice(["ring", "aerial"])
    c = dict(kind=kind, layout=layout, groups=0)
    if layout == "ring":
        c.update(cameras=_log(rng, 10, 80), points=_log(rng, 1_000, 60_000), views=rng.randint(4, 8))
    else:
        c.update(cameras=_log(rng, 36, 120 if kind == "schur" else 300), points=_log(rng, 4_000, 120_000),
                 views=rng.randint(6, 10))
    if kind == "backward":
        c.update(cameras=min(c["cameras"], 80), points=min(c["points"], 24_000), mixed=True)
        return c
    c.update(mixed=rng.random() < 0.6, damping=rng.choice([1e-4, 1e-3, 1e-2, 1e-1]))
    c["groups"] = rng.choice([0, 1, 2]) if layout == "aerial" else 0
    if kind == "step":
        c["trials"] = rng.choice([1, 1, 2, 8])
        if c["groups"]:  # (an undamped self-calibrating system is solved to a part in a million only)
            c["damping"] = max(1e-3, c["damping"])
    return c


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=F64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _rodrigues(w):
    """Rotation matrices exp([w]x) of vectors w [n, 3]."""
    th = w.norm(dim=1).clamp_min(1e-15)[:, None, None]
    K = torch.zeros(w.shape[0], 3, 3, device=w.device, dtype=w.dtype)
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 0] = -w[:, 2], w[:, 1], w[:, 2]
    K[:, 1, 2], K[:, 2, 0], K[:, 2, 1] = -w[:, 0], -w[:, 1], w[:, 0]
    K = K / th
    return torch.eye(3, device=w.device, dtype=w.dtype) + torch.sin(th) * K + (1 - torch.cos(th)) * (K @ K)


def _pixels(R, C, K, X):
    """Brown-Conrady pixels and depth of points X [..., 3]; K = fx, fy, cx, cy, k1, k2, k3, p1, p2."""
    d = X - C
    xc = (R * d[..., :, None]).sum(-2)
    z = xc[..., 2]
    x, y = xc[..., 0] / z, xc[..., 1] / z
    r2 = x * x + y * y
    rad = 1 + r2 * (K[..., 4] + r2 * (K[..., 5] + r2 * K[..., 6]))
    p1, p2 = K[..., 7], K[..., 8]
    xd = x * rad + 2 * p1 * x * y + p2 * (r2 + 2 * x * x)
    yd = y * rad + p1 * (r2 + 2 * y * y) + 2 * p2 * x * y
    return K[..., 0] * xd + K[..., 2], K[..., 1] * yd + K[..., 3], z


def _true_cameras(c):
    """True rotations, centres, calibrations and groups of the layout's cameras, and its frame."""
    nc = c["cameras"]
    if c["layout"] == "ring":
        a = 2 * math.pi * torch.arange(nc, device=DEV, dtype=F64) / nc
        C = torch.stack([10 * torch.cos(a), 10 * torch.sin(a), torch.full_like(a, 2.0)], 1)
        f = -C / C.norm(dim=1, keepdim=True)
        up = torch.tensor([0.0, 0.0, 1.0], device=DEV, dtype=F64).expand(nc, 3)
        r = torch.linalg.cross(f, up)
        r = r / r.norm(dim=1, keepdim=True)
        R = torch.stack([r, torch.linalg.cross(f, r), f], 2)
        K = torch.tensor([3500.0, 3500.0, 2000.0, 1500.0, -0.05, 0.01, 0.0, 1e-4, 1e-4], device=DEV,
                         dtype=F64).repeat(nc, 1)
        return R, C, K, torch.zeros(nc, device=DEV, dtype=torch.long), 4000.0, 3000.0
    along = max(2, int(round(math.sqrt(1.25 * nc))))
    i = torch.arange(nc, device=DEV)
    line, j = i // along, i % along
    # 100 m above ground, f = 4000 px, 6000 x 4000 px: 150 m x 100 m footprint, 80 % / 60 % overlap
    C = torch.stack([line * 60.0, j * 20.0, torch.full((nc,), 100.0, device=DEV)], 1).to(F64)
    R = torch.tensor([[1.0, 0, 0], [0, -1.0, 0], [0, 0, -1.0]], device=DEV, dtype=F64).repeat(nc, 1, 1)
    ng = max(1, c.get("groups", 0))
    g = line % ng
    K = torch.tensor([4000.0, 4000.0, 3000.0, 2000.0, -0.04, 0.008, -0.001, 1e-4, -1e-4], device=DEV,
                     dtype=F64).repeat(nc, 1)
    K[:, 0] *= 1 + 0.002 * g
    K[:, 1] = K[:, 0]
    K[:, 2] += 3.0 * g
    K[:, 3] -= 2.0 * g
    K[:, 4] += 0.005 * g
    return R, C, K, g, 6000.0, 4000.0


def _terrain(g):
    """Sum of eight sinusoids, 20 m: wave vectors, phases, amplitudes."""
    k = (0.003 + 0.027 * _rand(g, 8, 2)) * torch.sign(_rand(g, 8, 2) - 0.5)
    ph, a = 2 * math.pi * _rand(g, 8), 0.5 + _rand(g, 8)
    return k, ph, 20.0 * a / a.sum()


def _true_points(c, g, n, C, terrain):
    if c["layout"] == "ring":
        return 4.0 * _rand(g, n, 3) - 2.0
    lo, hi = C.min(0).values, C.max(0).values
    x = lo[0] - 10 + (hi[0] - lo[0] + 20) * _rand(g, n)
    y = lo[1] - 5 + (hi[1] - lo[1] + 10) * _rand(g, n)
    k, ph, a = terrain
    z = (a * torch.sin(x[:, None] * k[:, 0] + y[:, None] * k[:, 1] + ph)).sum(1)
    return torch.stack([x, y, z], 1)


def _scene(c, seed):
    """Cameras (true and initial), points, observations in track order, all float64 on the device.
    Whole solves start from raw matches, wrong ones anywhere in the frame (the initial-error gate
    drops their tracks); single steps from matches that passed a geometric check, wrong ones off by
    tens of pixels (every track takes part)."""
    g = _gen(seed)
    R, C, K, grp, width, height = _true_cameras(c)
    nc, n, most = R.shape[0], c["points"], c["views"]
    # views per point: 3 to c["views"] in equal shares, of the cameras that see it
    want = (3 + torch.arange(n, device=DEV) % (most - 2))[torch.randperm(n, generator=g, device=DEV)]
    ground = _terrain(g)
    kept, views, have, tries = [], [], 0, 0
    batch = max(1_000, min(n + n // 2, 8_000_000 // nc))
    while have < n:
        tries += 1
        if tries > 60 * (1 + n // batch):
            raise RuntimeError("too few points are seen by %d cameras" % most)
        X = _true_points(c, g, batch, C, ground)
        u, v, z = _pixels(R[None], C[None], K[None], X[:, None, :])
        seen = (z > 0.1) & (u >= 0) & (u < width) & (v >= 0) & (v < height)
        if c["layout"] != "ring":  # (the distortion polynomial folds far points back into the frame)
            d = (X[:, None, :2] - C[None, :, :2]).abs()
            seen &= (d[..., 0] < 90) & (d[..., 1] < 60)
        top, idx = torch.where(seen, _rand(g, batch, nc), -1.0).topk(most, dim=1)
        good = torch.nonzero(top[:, -1] >= 0)[:n - have, 0]
        kept.append(X[good])
        views.append(idx[good])
        have += good.numel()
    X, idx = torch.cat(kept), torch.cat(views)
    idx = torch.where(torch.arange(most, device=DEV)[None] < want[:, None], idx, nc).sort(1).values
    cam, trk = idx[idx < nc], torch.arange(n, device=DEV)[:, None].expand_as(idx)[idx < nc]
    u, v, _ = _pixels(R[cam], C[cam], K[cam], X[trk])
    no = cam.numel()
    u, v = u + 0.5 * _randn(g, no), v + 0.5 * _randn(g, no)
    wild = _rand(g, no) < (0.02 if c["layout"] == "ring" else 0.03)
    if c["kind"] in ("solve", "backward"):
        u = torch.where(wild, width * _rand(g, no), u)
        v = torch.where(wild, height * _rand(g, no), v)
    else:
        u = u + torch.where(wild, 20.0, 0.0) * _randn(g, no)
        v = v + torch.where(wild, 20.0, 0.0) * _randn(g, no)
    K0 = K.clone()
    if c.get("groups", 0) > 0:  # self-calibration starts from the maker's values
        K0[:] = torch.tensor([4000.0, 4000.0, 3000.0, 2000.0, 0.0, 0.0, 0.0, 0.0, 0.0], device=DEV, dtype=F64)
        K0[:, 4:9] = 0.9 * K[:, 4:9]
        for q in range(9):  # one start per group
            K0[:, q] = torch.stack([K0[grp == k][0, q] for k in range(int(grp.max()) + 1)])[grp]
    R0 = _rodrigues(0.003 * _randn(g, nc, 3)) @ R
    C0 = C + 0.05 * _randn(g, nc, 3)
    X0 = X + 0.05 * _randn(g, *X.shape)
    off = torch.cat([torch.zeros(1, device=DEV, dtype=torch.long), want.cumsum(0)])
    return dict(R=R0, C=C0, K=K0, X=X0, C_true=C, group=grp, cam=cam, trk=trk, u=u, v=v, off=off, width=width,
                height=height)


def _records(R, C, K, width, height):
    rec = torch.zeros(R.shape[0], 32, device=R.device, dtype=F64)
    rec[:, 0:9], rec[:, 9:12], rec[:, 12:21] = R.reshape(-1, 9), C, K
    rec[:, 21:26] = torch.tensor([1.0, 1.0, 0.0, width, height], device=R.device, dtype=F64)
    return rec


def _problem(c, sc):
    def host(t, dt):
        return np.ascontiguousarray(t.cpu().numpy().astype(dt))
    no = sc["cam"].numel()
    return Problem(cameras=host(_records(sc["R"], sc["C"], sc["K"], sc["width"], sc["height"]), np.float64),
                   points=host(sc["X"], np.float64), track_offsets=host(sc["off"], np.int64),
                   obs_camera=host(sc["cam"], np.int32), obs_u=host(sc["u"], np.float64),
                   obs_v=host(sc["v"], np.float64), obs_weight=np.ones(no), obs_scale=np.ones(no),
                   cameraCalibrationGroupIds=host(sc["group"], np.int32) if c.get("groups", 0) > 0 else None)


def _options(c):
    o = SolveOptions()
    o.solver.imageRobustLoss = ImageRobustLoss.Huber if c["layout"] == "ring" else ImageRobustLoss.Cauchy
    o.solver.imageRobustLossScalePixels = 1.5
    o.solver.maxIterations = 50 if c["kind"] == "rig" else 40
    o.backend.enablePlaMatrixMixedPrecision = bool(c["mixed"])
    if c.get("groups", 0) > 0:
        o.calibration.refineSharedFocalLength = True
        o.calibration.refineSharedPrincipalPoint = True
        o.calibration.refineSharedRadialDistortion = True
    return o


def _ok(status, what):
    if status != 0:
        raise RuntimeError("%s returned status %d" % (what, status))


def _targets(sc, seed):
    """Surveyed camera centres for the loss of the backward pass."""
    return sc["C_true"] + 0.1 * _randn(_gen(seed + 77_777), sc["C_true"].shape[0], 3)


def _objective_inputs(c, seed):
    g = _gen(seed)
    R, C, K, _, width, height = _true_cameras(c)
    n, nc, npt = c["observations"], c["cameras"], c["points"]
    X = _true_points(c, g, npt, C, _terrain(g))
    pt = torch.arange(n, device=DEV) * npt // n
    if c["layout"] == "ring":
        cam = torch.randint(0, nc, (n,), generator=g, device=DEV)
    else:  # one of the four nearest cameras on the ground
        near = torch.cat([torch.cdist(X[s:s + 50_000, :2], C[:, :2]).topk(4, dim=1, largest=False).indices
                          for s in range(0, npt, 50_000)])
        cam = near[pt, torch.randint(0, 4, (n,), generator=g, device=DEV)]
    u, v, _ = _pixels(R[cam], C[cam], K[cam], X[pt])
    wild = _rand(g, n) < 0.03
    u = torch.where(wild, width * _rand(g, n), u + 0.5 * _randn(g, n))
    v = torch.where(wild, height * _rand(g, n), v + 0.5 * _randn(g, n))
    R0 = _rodrigues(0.001 * _randn(g, nc, 3)) @ R
    return dict(cams=_records(R0, C, K, width, height).contiguous(), X=(X + 0.02 * _randn(g, npt, 3)).contiguous(),
                cam=cam.to(torch.int32).contiguous(), pt=pt.to(torch.int32).contiguous(), u=u, v=v,
                w=torch.ones(n, device=DEV, dtype=F64), loss=1 if c["layout"] == "ring" else 2)


def _equations(c, seed):
    """Residual blocks of a host assembly: two primary blocks of 13 columns may share a residual."""
    rng = np.random.default_rng(seed)
    P, E, v = c["blocks"], c["eliminated"], min(c["views"], c["blocks"])
    prim = np.sort(np.argsort(rng.random((E, P)), axis=1)[:, :v], axis=1)
    n = E * v
    return dict(prim=prim.reshape(-1).astype(np.int32), elim=np.repeat(np.arange(E), v),
                Jp=rng.normal(size=(n, 2, 13)) * 0.5, Je=rng.normal(size=(n, 2, 3)), r=rng.normal(size=(n, 2)) * 0.1,
                w=rng.uniform(0.5, 1.5, n), prior=rng.uniform(0.5, 1.5, P))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "objective":
        s = _objective_inputs(case, seed)
        return dict(case=case, lib=native.load(), **s)
    if kind == "blockschur":
        q = _equations(case, seed)
        eq = BlockNormalEquations(case["blocks"], case["eliminated"], 13, 3)
        for i in range(q["r"].shape[0]):
            eq.addResidualBlocks([q["prim"][i]], [q["Jp"][i]], int(q["elim"][i]), q["Je"][i], q["r"][i], q["w"][i])
        eye = np.eye(13)
        for b in range(case["blocks"]):
            eq.addPrimaryResidualBlock(b, q["prior"][b] * eye, np.zeros(13))
        return dict(case=case, eq=eq, ctx=Gb300Context(0),
                    opt=SchurComplementSolverOptions(useMixedPrecision=bool(case["mixed"])))
    if kind == "rig":
        lines = 3
        p = synth.rig_grid_problem(seed=seed, n_along=max(2, case["cameras"] // (5 * lines)), n_lines=lines,
                                   n_points=case["points"], max_views=case["views"])
        synth.with_control_points(p, n=12, sigma=0.02, seed=seed + 1)
        synth.with_scale_bars(p, n=4, sigma=0.005, seed=seed + 2)
        return dict(case=case, problem=p, options=_options(case), solver=Solver(), ws=SolverWorkspace(0))
    sc = _scene(case, seed)
    p, o = _problem(case, sc), _options(case)
    if kind == "solve":
        return dict(case=case, problem=p, options=o, solver=Solver(), ws=SolverWorkspace(0))
    ctx = Gb300Context(0)
    _ok(ctx.upload(p, o), "upload")
    if kind == "backward":
        ctx.solve()
        newton_polish(ctx, iterations=4)
        d = ctx.download()["cameras"][:, 9:12] - _targets(sc, seed).cpu().numpy()
        grad = np.zeros((p.n_cameras, 6))
        grad[:, 3:6] = 2.0 * d
        return dict(case=case, ctx=ctx, grad=grad)
    precision = Precision.Mixed if case["mixed"] else Precision.Fp64
    ctx.linearize_schur(case["damping"], precision)  # the plan is built with the first linearisation
    return dict(case=case, ctx=ctx, precision=precision, damping=case["damping"],
                alphas=[2.0 ** -k for k in range(case.get("trials", 1))])


def run(state):
    kind = state["case"]["kind"]
    if kind == "objective":
        s = state
        cost, bad = ctypes.c_double(0.0), ctypes.c_int64(0)
        stream = torch.cuda.current_stream().cuda_stream
        _ok(s["lib"].pb_gpu_objective_noalloc(
            s["cams"].data_ptr(), s["cams"].shape[0], s["X"].data_ptr(), s["X"].shape[0], s["cam"].data_ptr(),
            s["pt"].data_ptr(), s["u"].data_ptr(), s["v"].data_ptr(), s["w"].data_ptr(), s["u"].numel(), s["loss"],
            1.5, stream, ctypes.byref(cost), ctypes.byref(bad)), "objective")
        return {"cost": cost.value, "invalid": int(bad.value)}
    if kind == "blockschur":
        x, y, _ = solve_damped_schur_complement(state["ctx"], state["eq"], state["case"]["damping"], state["opt"])
        return {"primary": x, "eliminated": y}
    if kind in ("solve", "rig"):
        r = state["solver"].solve(state["problem"], state["options"], state["ws"])
        return {"cameras": r.refinedCameras, "points": r.points.point, "valid": r.points.valid}
    ctx = state["ctx"]
    if kind == "backward":
        out = ctx.backward(grad_cameras=state["grad"])
        return {"observations": out["observations"], "initial_cameras": out["initial_cameras"]}
    cost, _ = ctx.linearize_schur(state["damping"], state["precision"])
    if kind == "schur":
        S, rhs, direct = ctx.reduced()
        return {"cost": cost, "matrix": S, "rhs": rhs, "direct": direct}
    step, _, _, _ = ctx.solve_reduced()
    points, decrease, _ = ctx.back_substitute()
    return {"cost": cost, "step": step, "points": points, "decrease": decrease,
            "trial_costs": ctx.cost_batch(state["alphas"])}


def work(case):
    kind = case["kind"]
    if kind == "objective":
        n = case["observations"]
        return {"bytes": 32 * n + 24 * case["points"] + 256 * case["cameras"], "flops": 90 * n}
    if kind == "blockschur":
        n, E, v = 13 * case["blocks"], case["eliminated"], case["views"]
        return {"bytes": 8 * (E * (v * 39 + 15) + 13 * n), "flops": E * v * v * 13 * 13 * 3 + n ** 3 / 3 + 2 * n * n}
    v = min(case["cameras"], (3 + case["views"]) / 2)
    no, nt, nc = case["points"] * v, case["points"], case["cameras"]
    nb = 8 * case.get("groups", 0)
    n = 6 * nc + nb
    inputs = 28 * no + 28 * nt + 256 * nc
    # linearisation, point blocks, pair blocks of every track, border and intrinsic block
    schur = no * 400 + nt * (v * (v + 1) / 2) * 36 * 6 + no * nb * 36 + nt * nb * nb * 6
    if kind == "schur":
        return {"bytes": inputs + 8 * n * n, "flops": schur}
    step = {"bytes": inputs + 24 * nt + 16 * n, "flops": schur + n ** 3 / 3 + 4 * n * n + no * 60 + no * 90}
    if kind == "step":
        return step
    if kind == "backward":
        return {"bytes": inputs + 16 * no, "flops": 3 * step["flops"]}
    # a whole solve: about ten steps
    return {"bytes": 10 * step["bytes"], "flops": 10 * step["flops"]}


# ---------------------------------------------------------------- 64-bit values in plain torch
class _Chart:
    """The block in the solver's chart: rotation increment D E(w)^T D R with E = Rx Ry Rz and D =
    diag(1, -1, -1), world centre (the scale camera: two tangent coordinates on the sphere around
    the anchor), point increment X + s(X) dX, additive calibration of the group."""

    def __init__(self, c, sc):
        self.c, self.loss, self.scale = c, 1 if c["layout"] == "ring" else 2, 1.5
        self.R, self.C, self.K, self.X = (sc[k].clone() for k in ("R", "C", "K", "X"))
        nc = self.C.shape[0]
        self.ng = c.get("groups", 0)
        self.ni = 8 if self.ng else 0
        self.group = sc["group"]
        u0, v0, z = _pixels(self.R[sc["cam"]], self.C[sc["cam"]], self.K[sc["cam"]], self.X[sc["trk"]])
        sq = (u0 - sc["u"]) ** 2 + (v0 - sc["v"]) ** 2
        nt = self.X.shape[0]
        tot = torch.zeros(nt, device=DEV, dtype=F64).index_add_(0, sc["trk"], torch.where(z > 1e-9, sq, math.inf))
        count = sc["off"][1:] - sc["off"][:-1]
        self.active = torch.sqrt(tot / (2 * count)) <= 100.0
        self.obs = self.active[sc["trk"]]
        self.cam, self.u, self.v = (sc[k][self.obs] for k in ("cam", "u", "v"))
        self.track_of = torch.cumsum(self.active, 0) - 1
        self.trk = self.track_of[sc["trk"][self.obs]]
        self.nt = int(self.active.sum())
        count = count[self.active]
        self.L = int(count.max())
        first = torch.cat([torch.zeros(1, device=DEV, dtype=torch.long), count.cumsum(0)[:-1]])
        self.place = self.trk * self.L + torch.arange(self.cam.numel(), device=DEV) - first[self.trk]
        # gauge: camera 0 fixed, the camera farthest from it keeps its distance
        d2 = ((self.C - self.C[0]) ** 2).sum(1)
        self.far = int(d2.argmax())
        self.base = math.sqrt(float(d2.max()))
        used = torch.zeros(nc, device=DEV, dtype=torch.bool)
        used[self.cam] = True
        used[0] = False
        self.block = torch.where(used, torch.cumsum(used, 0) - 1, -1)
        self.ncb = int(used.sum())
        self.nb = self.ng * self.ni
        self.n = 6 * self.ncb + self.nb
        self.params = torch.stack([self.K[self.group == k][0] for k in range(max(1, self.ng))])
        self.prior = self.params.clone()
        f = self.prior[:, 0]
        one = torch.ones_like(f)
        self.inv_sigma = torch.stack([1 / (0.35 * f), 1 / (0.04 * f), 1 / (0.04 * f), one / 0.15, one / 0.15,
                                      one / 0.15, one / 0.01, one / 0.01], 1)
        self.tracks_in = torch.nonzero(self.active)[:, 0]

    COLS = [0, 2, 3, 4, 5, 6, 7, 8]

    def basis(self):
        """World-frame tangent directions of the scale camera's sphere."""
        D = torch.tensor([1.0, -1.0, -1.0], device=DEV, dtype=F64)
        u = D * (self.C[self.far] - self.C[0])
        u = u / u.norm()
        a = u.abs()
        axis = 1 if a[0] > a[1] else 0
        if a[axis] > a[2]:
            axis = 2
        e = torch.zeros(3, device=DEV, dtype=F64)
        e[axis] = 1.0
        s = torch.linalg.cross(e, u)
        s = s / s.norm()
        return torch.stack([D * torch.linalg.cross(u, s), D * s])

    def calibration(self):
        return self.params[self.group] if self.ng else self.K

    def scales(self):
        ln = self.X[self.active].norm(dim=1) / 1000.0
        return torch.where(ln > 0, ln / torch.atan(ln), torch.ones_like(ln))

    def data(self):
        cam, K = self.cam, self.calibration()
        s = self.scales()[self.trk]
        return (self.R[cam], self.C[cam], K[cam], self.X[self.active][self.trk], s, (cam == self.far).to(F64), self.u,
                self.v)

    def residual(self, gb, anchor):
        base = self.base

        def f(z, R, C, K, X, s, tangent, u, v):
            sn, cs = torch.sin(z[:3]), torch.cos(z[:3])
            one, zero = torch.ones_like(sn[0]), torch.zeros_like(sn[0])
            Rx = torch.stack([one, zero, zero, zero, cs[0], -sn[0], zero, sn[0], cs[0]]).reshape(3, 3)
            Ry = torch.stack([cs[1], zero, sn[1], zero, one, zero, -sn[1], zero, cs[1]]).reshape(3, 3)
            Rz = torch.stack([cs[2], -sn[2], zero, sn[2], cs[2], zero, zero, zero, one]).reshape(3, 3)
            D = torch.tensor([1.0, -1.0, -1.0], device=z.device, dtype=F64)
            Rn = (D[:, None] * (Rx @ Ry @ Rz).T * D[None]) @ R
            e = C + z[3] * gb[0] + z[4] * gb[1] - anchor + (1 - tangent)  # (no zero vector at the anchor)
            Cn = tangent * (anchor + base * e / torch.sqrt((e * e).sum())) + (1 - tangent) * (C + z[3:6])
            Kn = K
            if z.shape[0] > 9:
                i = z[9:]
                fx = K[0] + i[0]
                Kn = torch.cat([torch.stack([fx, fx * (K[1] / K[0])]), K[2:] + i[1:]])
            pu, pv, _ = _pixels(Rn, Cn, Kn, X + s * z[6:9])
            return torch.stack([pu - u, pv - v])
        return f

    def rho(self, sq):
        c2 = self.scale ** 2
        if self.loss == 1:
            n = torch.sqrt(torch.where(sq > c2, sq, c2))
            return torch.where(sq <= c2, 0.5 * sq, self.scale * n - 0.5 * c2)
        return 0.5 * c2 * torch.log1p(sq / c2)

    def weight(self, sq):
        c2 = self.scale ** 2
        if self.loss == 1:
            return torch.where(sq <= c2, torch.ones_like(sq), self.scale / torch.sqrt(sq.clamp_min(c2)))
        return 1 / (1 + sq / c2)

    def cost(self, R=None, C=None, params=None, X=None):
        R, C = self.R if R is None else R, self.C if C is None else C
        params = self.params if params is None else params
        K = params[self.group] if self.ng else self.K
        X = self.X[self.active] if X is None else X
        u, v, _ = _pixels(R[self.cam], C[self.cam], K[self.cam], X[self.trk])
        total = self.rho((u - self.u) ** 2 + (v - self.v) ** 2).sum()
        if self.ng:
            total = total + 0.5 * ((self.inv_sigma * (params - self.prior)[:, self.COLS]) ** 2).sum()
        return float(total)

    def padded(self, a):
        out = torch.zeros(self.nt * self.L, *a.shape[1:], device=DEV, dtype=a.dtype)
        out[self.place] = a
        return out.reshape(self.nt, self.L, *a.shape[1:])

    def batched(self, f, gb, most):
        """f(z, observation) at z = 0 over all observations, `most` at a time."""
        data, z = self.data(), torch.zeros(9 + self.ni, device=DEV, dtype=F64)
        g = torch.func.vmap(f, in_dims=(None,) + (0,) * 8)
        n = self.cam.numel()
        return torch.cat([g(z, *(d[s:s + most] for d in data)) for s in range(0, n, most)])

    def normal(self, exact_hessian=False):
        """Per observation: Hessian (9 + ni)^2 and -gradient, Gauss-Newton or exact."""
        gb, anchor = self.basis(), self.C[0]
        res = self.residual(gb, anchor)
        gb.requires_grad_(False)
        J = self.batched(torch.func.jacfwd(res), gb, 200_000)
        r = self.batched(res, gb, 200_000)
        w = self.weight((r * r).sum(1))
        g = -(J * (w[:, None] * r)[..., None]).sum(1)
        if exact_hessian:
            def one(z, *a):
                q = res(z, *a)
                return self.rho((q * q).sum())
            H = self.batched(torch.func.hessian(one), gb, 25_000)
        else:
            H = (w[:, None, None, None] * J[..., :, None] * J[..., None, :]).sum(1)
        tg = self.cam == self.far
        return H, g, J, r, w, tg

    def reduce(self, H, g, damping, bp=None):
        """Point elimination: the reduced matrix, its right-hand side, the direct one, and what the
        back-substitution needs.  bp: another right-hand side of the points."""
        b, ncb, ni, ng, n6 = self.block[self.cam], self.ncb, self.ni, self.ng, 6 * self.ncb
        Hp, gp = self.padded(H), self.padded(g)
        blk = self.padded(b + 1) - 1
        grp = self.padded(self.group[self.cam] + 1) - 1
        V = Hp[..., 6:9, 6:9].sum(1)
        V = V + damping * torch.diag_embed(torch.diagonal(V, dim1=1, dim2=2))
        Vi = torch.linalg.inv(V)
        q = gp[..., 6:9].sum(1) if bp is None else bp
        W = Hp[..., 0:6, 6:9]
        S4 = torch.zeros((ncb + 1) * (ncb + 1), 36, device=DEV, dtype=F64)
        dst = torch.where(blk >= 0, blk, ncb)
        S4.index_add_(0, (dst * (ncb + 1) + dst).reshape(-1), Hp[..., 0:6, 0:6].reshape(-1, 36))
        step = max(1, 2_000_000 // (self.L * self.L))
        for s in range(0, self.nt, step):
            Y = W[s:s + step] @ Vi[s:s + step, None]
            P = torch.einsum("tiak,tjbk->tijab", Y, W[s:s + step]).reshape(-1, 36)
            d = dst[s:s + step]
            S4.index_add_(0, (d[:, :, None] * (ncb + 1) + d[:, None, :]).reshape(-1), -P)
        S = torch.zeros(self.n, self.n, device=DEV, dtype=F64)
        S[:n6, :n6] = S4.reshape(ncb + 1, ncb + 1, 6, 6)[:ncb, :ncb].permute(0, 2, 1, 3).reshape(n6, n6)
        rhs6 = torch.zeros(ncb + 1, 6, device=DEV, dtype=F64)
        dir6 = torch.zeros(ncb + 1, 6, device=DEV, dtype=F64)
        dir6.index_add_(0, dst.reshape(-1), gp[..., 0:6].reshape(-1, 6))
        Vq = (Vi @ q[..., None])[..., 0]
        rhs6.index_add_(0, dst.reshape(-1), -(W @ Vq[:, None, :, None])[..., 0].reshape(-1, 6))
        rhs = torch.zeros(self.n, device=DEV, dtype=F64)
        direct = torch.zeros(self.n, device=DEV, dtype=F64)
        direct[:n6] = dir6[:ncb].reshape(-1)
        rhs[:n6] = rhs6[:ncb].reshape(-1)
        Kt = None
        if ng:
            hot = torch.nn.functional.one_hot(grp.clamp_min(0), ng).to(F64) * (grp >= 0)[..., None]
            Kt = torch.einsum("tlg,tlck->tgck", hot, Hp[..., 9:, 6:9]).reshape(self.nt, self.nb, 3)
            KV = Kt @ Vi
            B = torch.einsum("tlac,tlg->tlagc", Hp[..., 0:6, 9:], hot).reshape(self.nt, self.L, 6, self.nb)
            B = B - W @ KV.transpose(1, 2)[:, None]
            Bs = torch.zeros(ncb + 1, 6 * self.nb, device=DEV, dtype=F64)
            Bs.index_add_(0, dst.reshape(-1), B.reshape(-1, 6 * self.nb))
            S[:n6, n6:] = Bs[:ncb].reshape(n6, self.nb)
            S[n6:, :n6] = S[:n6, n6:].T
            Hkk = torch.einsum("tlcd,tlg->gcd", Hp[..., 9:, 9:], hot)
            S[n6:, n6:] = torch.block_diag(*Hkk) - torch.einsum("tak,tbk->ab", KV, Kt)
            direct[n6:] = torch.einsum("tlc,tlg->gc", gp[..., 9:], hot).reshape(-1)
            rhs[n6:] = -torch.einsum("tak,tk->a", Kt, Vq)
            off = (self.inv_sigma ** 2 * (self.params - self.prior)[:, self.COLS]).reshape(-1)
            direct[n6:] -= off
            S[n6:, n6:] += torch.diag((self.inv_sigma ** 2).reshape(-1))
        rhs = rhs + direct
        dg = torch.diagonal(S)
        S[range(self.n), range(self.n)] = torch.where(dg != 0, dg * (1 + damping), torch.ones_like(dg))
        return S, rhs, direct, (Vi, q, W, Kt, dst)

    def points_of(self, x, back):
        Vi, q, W, Kt, dst = back
        x6 = torch.cat([x[:6 * self.ncb].reshape(self.ncb, 6), torch.zeros(1, 6, device=DEV, dtype=F64)])
        t = (W * x6[dst][..., None]).sum((1, 2))
        if Kt is not None:
            t = t + torch.einsum("tak,a->tk", Kt, x[6 * self.ncb:])
        return (Vi @ (q - t)[..., None])[..., 0]

    def moved(self, x, dp, alpha):
        """State after alpha times the step (x, dp)."""
        z = torch.zeros(self.C.shape[0], 6, device=DEV, dtype=F64)
        z[self.block >= 0] = x[:6 * self.ncb].reshape(self.ncb, 6)
        z = alpha * z
        sn, cs = torch.sin(z[:, :3]), torch.cos(z[:, :3])
        E = torch.eye(3, device=DEV, dtype=F64).repeat(z.shape[0], 1, 1)
        for a, (i, j) in enumerate(((1, 2), (2, 0), (0, 1))):
            G = torch.eye(3, device=DEV, dtype=F64).repeat(z.shape[0], 1, 1)
            G[:, i, i] = G[:, j, j] = cs[:, a]
            G[:, i, j], G[:, j, i] = -sn[:, a], sn[:, a]
            E = E @ G
        D = torch.tensor([1.0, -1.0, -1.0], device=DEV, dtype=F64)
        R = (D[:, None] * E.transpose(1, 2) * D) @ self.R
        C = self.C + z[:, 3:]
        gb = self.basis()
        e = self.C[self.far] + z[self.far, 3] * gb[0] + z[self.far, 4] * gb[1] - self.C[0]
        C[self.far] = self.C[0] + self.base * e / e.norm()
        X = self.X[self.active] + alpha * self.scales()[:, None] * dp
        params = self.params.clone()
        if self.ng:
            d = alpha * x[6 * self.ncb:].reshape(self.ng, self.ni)
            asp = params[:, 1] / params[:, 0]
            params[:, self.COLS] += d
            params[:, 1] = params[:, 0] * asp
        return R, C, params, X

    def take(self, state):
        self.R, self.C, self.params, X = state
        self.X[self.active] = X

    def fixed_point(self):
        """Gauss-Newton steps with halving, then exact Newton steps."""
        cost = self.cost()
        for it in range(60):
            H, g, *_ = self.normal()
            S, rhs, _, back = self.reduce(H, g, 0.0)
            x = _solve(S, rhs)
            dp = self.points_of(x, back)
            alpha, moved = 1.0, False
            for _ in range(12):
                state = self.moved(x, dp, alpha)
                trial = self.cost(*state)
                if trial < cost:
                    moved = True
                    break
                alpha /= 2
            if not moved:
                break
            self.take(state)
            cost = trial
            if alpha * float(x.abs().max()) < 1e-5:
                break
        for _ in range(4):
            H, g, *_ = self.normal(True)
            S, rhs, _, back = self.reduce(H, g, 0.0)
            x = _solve(S, rhs)
            self.take(self.moved(x, self.points_of(x, back), 1.0))


def _solve(S, b):
    d = torch.rsqrt(torch.diagonal(S).abs())
    A = S * d[:, None] * d
    LU = torch.linalg.lu_factor(A)
    x = torch.linalg.lu_solve(*LU, (d * b)[:, None])
    x = x + torch.linalg.lu_solve(*LU, (d * b)[:, None] - A @ x)
    return d * x[:, 0]


def _exact_objective(c, seed):
    s = _objective_inputs(c, seed)
    rec, cam = s["cams"], s["cam"].long()
    R, C, K = rec[:, 0:9].reshape(-1, 3, 3), rec[:, 9:12], rec[:, 12:21]
    total, bad = 0.0, 0
    for a in range(0, cam.numel(), 500_000):
        k, p = cam[a:a + 500_000], s["pt"][a:a + 500_000].long()
        u, v, z = _pixels(R[k], C[k], K[k], s["X"][p])
        sq = (u - s["u"][a:a + 500_000]) ** 2 + (v - s["v"][a:a + 500_000]) ** 2
        if s["loss"] == 1:
            rho = torch.where(sq <= 2.25, 0.5 * sq, 1.5 * torch.sqrt(sq) - 1.125)
        else:
            rho = 1.125 * torch.log1p(sq / 2.25)
        good = z > 1e-9
        total += float(rho[good].sum())
        bad += int((~good).sum())
    return {"cost": total, "invalid": bad}


def _exact_blockschur(c, seed):
    q = _equations(c, seed)
    P, E, lam = c["blocks"], c["eliminated"], c["damping"]
    n = 13 * P
    Jp, Je, r, w = (torch.from_numpy(q[k]).to(DEV) for k in ("Jp", "Je", "r", "w"))
    prim, elim = torch.from_numpy(q["prim"]).to(DEV).long(), torch.from_numpy(q["elim"]).to(DEV).long()
    v = prim.numel() // E
    Hpp = torch.zeros(P, 13, 13, device=DEV, dtype=F64)
    Hpp.index_add_(0, prim, torch.einsum("n,nra,nrb->nab", w, Jp, Jp))
    Hpp += torch.diag_embed(torch.from_numpy(q["prior"]).to(DEV)[:, None].expand(P, 13) ** 2)
    gp = torch.zeros(P, 13, device=DEV, dtype=F64).index_add_(0, prim, torch.einsum("n,nra,nr->na", w, Jp, r))
    V = torch.zeros(E, 3, 3, device=DEV, dtype=F64).index_add_(0, elim, torch.einsum("n,nra,nrb->nab", w, Je, Je))
    ge = torch.zeros(E, 3, device=DEV, dtype=F64).index_add_(0, elim, torch.einsum("n,nra,nr->na", w, Je, r))
    V = V + lam * torch.diag_embed(torch.diagonal(V, dim1=1, dim2=2))
    Hpp = Hpp + lam * torch.diag_embed(torch.diagonal(Hpp, dim1=1, dim2=2))
    Vi = torch.linalg.inv(V)
    W = torch.einsum("n,nra,nrb->nab", w, Jp, Je).reshape(E, v, 13, 3)
    pr = prim.reshape(E, v)
    S = torch.zeros(P * P, 169, device=DEV, dtype=F64)
    S.index_add_(0, torch.arange(P, device=DEV) * (P + 1), Hpp.reshape(P, 169))
    S.index_add_(0, (pr[:, :, None] * P + pr[:, None, :]).reshape(-1),
                 -torch.einsum("eiak,ekl,ejbl->eijab", W, Vi, W).reshape(-1, 169))
    S = S.reshape(P, P, 13, 13).permute(0, 2, 1, 3).reshape(n, n)
    b = -gp
    b = b.index_add(0, prim, torch.einsum("eiak,ekl,el->eia", W, Vi, ge).reshape(-1, 13)).reshape(n)
    x = _solve(S, b)
    y = torch.einsum("ekl,el->ek", Vi, -ge - torch.einsum("eiak,eia->ek", W, x.reshape(P, 13)[pr]))
    return {"primary": x.cpu().numpy(), "eliminated": y.reshape(-1).cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "objective":
        return _exact_objective(case, seed)
    if kind == "blockschur":
        return _exact_blockschur(case, seed)
    if kind in ("solve", "rig"):
        return None  # the stopping rule ends the iterations short of the minimum: no closed form
    sc = _scene(case, seed)
    m = _Chart(case, sc)
    if kind == "backward":
        m.fixed_point()
        H, g, J, r, w, _ = m.normal(True)
        bc = torch.zeros(m.C.shape[0], 6, device=DEV, dtype=F64)
        bc[:, 3:] = 2 * (m.C - _targets(sc, seed))
        gb = m.basis()
        t = bc[m.far, 3:].clone()
        bc[m.far, 3:] = torch.stack([t @ gb[0], t @ gb[1], torch.zeros((), device=DEV, dtype=F64)])
        zero = torch.zeros(m.nt, 3, device=DEV, dtype=F64)
        S, _, _, back = m.reduce(H, torch.zeros_like(g), 0.0, bp=zero)
        b = torch.zeros(m.n, device=DEV, dtype=F64)
        b[:6 * m.ncb] = bc[m.block >= 0].reshape(-1)
        mu = _solve(S, b)
        mp = m.points_of(mu, back)
        # d2F / dz d(u, v) = -J^T W2: dL/d(u, v) = W2 J mu
        z = torch.zeros(m.cam.numel(), 9 + m.ni, device=DEV, dtype=F64)
        x6 = torch.cat([mu[:6 * m.ncb].reshape(m.ncb, 6), torch.zeros(1, 6, device=DEV, dtype=F64)])
        z[:, :6] = x6[torch.where(m.block >= 0, m.block, m.ncb)[m.cam]]
        z[:, 6:9] = mp[m.trk]
        if m.ng:
            z[:, 9:] = mu[6 * m.ncb:].reshape(m.ng, m.ni)[m.group[m.cam]]
        Jm = (J * z[:, None, :]).sum(2)
        sq = (r * r).sum(1)
        c2 = m.scale ** 2
        if m.loss == 1:  # rho' = 1/2 min(1, c / |r|)
            d2 = torch.where(sq <= c2, torch.zeros_like(sq), -0.25 * m.scale / sq.clamp_min(c2) ** 1.5)
        else:
            d2 = -0.5 / (1 + sq / c2) ** 2 / c2
        out = torch.zeros(sc["cam"].numel(), 2, device=DEV, dtype=F64)
        out[m.obs] = w[:, None] * Jm + 4 * d2[:, None] * (r * Jm).sum(1, keepdim=True) * r
        return {"observations": out.cpu().numpy(), "initial_cameras": None}
    H, g, *_ = m.normal()
    S, rhs, direct, back = m.reduce(H, g, case["damping"])
    if kind == "schur":
        return {"cost": m.cost(), "matrix": S.cpu().numpy(), "rhs": rhs.cpu().numpy(), "direct": direct.cpu().numpy()}
    x = _solve(S, rhs)
    dp = m.points_of(x, back)
    dd = float(direct @ x + (back[1] * dp).sum())
    costs = [m.cost(*m.moved(x, dp, 2.0 ** -k)) for k in range(case["trials"])]
    return {"cost": m.cost(), "step": x.cpu().numpy(), "points": dp.reshape(-1).cpu().numpy(), "decrease": dd,
            "trial_costs": np.array(costs)}
