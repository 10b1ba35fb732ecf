"""Fixed workloads for profiling the backend under ncu.

    python -m plabundle_gb300.profile_case --workload aerial500 --precision mixed --iterations 3
    python -m plabundle_gb300.profile_case --workload aerial250 --precision mixed --iterations 3
    python -m plabundle_gb300.profile_case --workload aerial250 --precision mixed --iterations 3 --linear-solver 2
    python -m plabundle_gb300.profile_case --workload aerial60 --precision fp64 --iterations 3
    python -m plabundle_gb300.profile_case --workload aerial60 --precision mixed --iterations 40 --backward
    python -m plabundle_gb300.profile_case --workload rig3000 --precision mixed --iterations 2
    python -m plabundle_gb300.profile_case --workload blockschur --precision fp64

`aerial500` is the 500-camera / 200k-point aerial grid of the benchmark (Cauchy 1.5 px, two
calibration groups refining f, cx, cy, k1-k3, p1, p2); `aerial250` the same generator at half
size (250 cameras, 100k points), small enough for `ncu --set full` captures; `aerial60` the generator
at 60 cameras and 20k points, whose reduced system (370 unknowns) one cluster solves; `rig3000` the oblique
rig block of the large survey configuration (600 five-camera rig captures, 1.5 M points, ~8 M
observations, 40 control points, 10 scale bars; general path).  `--backward` adds a backward pass of the
solved state.  `blockschur` is the damped Schur solve of 40 primary blocks of 13 columns and 3 000
eliminated ones, twice.  Otherwise one LM iteration is
solved first on a separate context (module loading, pattern build), then the profiled solve of
`--iterations` iterations.
"""
from __future__ import annotations

import argparse

import numpy as np

from . import synth
from .device import Gb300Context
from .problem import ImageRobustLoss, SolveOptions
from .schur import BlockNormalEquations, SchurComplementSolverOptions, solve_damped_schur_complement


def workload(name: str, mixed: bool, iterations: int):
    if name == "rig3000":
        p = synth.rig_grid_problem(seed=21)
        synth.with_control_points(p, n=40, sigma=0.02, seed=3)
        synth.with_scale_bars(p, n=10, sigma=0.005, seed=5)
        o = SolveOptions()
        o.solver.imageRobustLoss = ImageRobustLoss.Cauchy
        o.solver.imageRobustLossScalePixels = 1.5
        o.backend.linearRelativeTolerance = 1e-6
        o.backend.enablePlaMatrixMixedPrecision = mixed
        o.solver.maxIterations = iterations
        return p, o
    if name == "aerial500":
        p = synth.aerial_grid_problem(seed=11)
    elif name == "aerial250":
        p = synth.aerial_grid_problem(seed=11, n_along=25, n_lines=10, n_points=100_000)
    elif name == "aerial60":
        p = synth.aerial_grid_problem(seed=11, n_along=10, n_lines=6, n_points=20_000)
    else:
        raise ValueError(name)
    o = SolveOptions()
    o.solver.imageRobustLoss = ImageRobustLoss.Cauchy
    o.solver.imageRobustLossScalePixels = 1.5
    o.calibration.refineSharedFocalLength = True
    o.calibration.refineSharedPrincipalPoint = True
    o.calibration.refineSharedRadialDistortion = True
    o.backend.enablePlaMatrixMixedPrecision = mixed
    o.solver.maxIterations = iterations
    return p, o


def block_schur(mixed: bool):
    rng = np.random.default_rng(7)
    eq = BlockNormalEquations(40, 3000, 13, 3)
    for b in range(40):
        eq.addPrimaryResidualBlock(b, np.eye(13), np.zeros(13))
    for e in range(3000):
        for b in np.sort(rng.choice(40, 5, replace=False)):
            eq.addResidualBlocks([int(b)], [rng.normal(size=(2, 13)) * 0.5], e, rng.normal(size=(2, 3)),
                                 rng.normal(size=2) * 0.1, rng.uniform(0.5, 1.5))
    ctx = Gb300Context(0)
    for _ in range(2):
        _, _, rep = solve_damped_schur_complement(ctx, eq, 1e-3, SchurComplementSolverOptions(useMixedPrecision=mixed))
    print("blockschur", "mixed" if mixed else "fp64", "converged", rep["converged"], "iterations", rep["iterations"])


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--workload", default="aerial250",
                    choices=["aerial60", "aerial250", "aerial500", "rig3000", "blockschur"])
    ap.add_argument("--precision", default="mixed", choices=["mixed", "fp64"])
    ap.add_argument("--iterations", type=int, default=3)
    ap.add_argument("--linear-solver", type=int, default=0, choices=[0, 1, 2],
                    help="0 automatic, 1 dense-factor-preconditioned CG, 2 block-Jacobi PCG")
    ap.add_argument("--backward", action="store_true", help="a backward pass of the solved state")
    a = ap.parse_args()
    mixed = a.precision == "mixed"
    if a.workload == "blockschur":
        block_schur(mixed)
        return
    p, o = workload(a.workload, mixed, 1)
    o.backend.linearSolver = a.linear_solver
    warm = Gb300Context(0)
    assert warm.upload(p, o) == 0
    warm.solve()
    warm.close()
    o.solver.maxIterations = a.iterations
    ctx = Gb300Context(0)
    assert ctx.upload(p, o) == 0
    rep = ctx.solve()
    print(a.workload, a.precision, "status", rep["status"], "iterations", rep["iterations"],
          "observations", p.n_obs, "final_cost", rep["final_cost"])
    if a.backward:
        out = ctx.backward(grad_cameras=np.ones((p.n_cameras, 6)))
        print("backward residual", out["report"]["relative_residual"])


if __name__ == "__main__":
    main()
