"""Small and odd-shaped runs of the sweep solvers, the reference's V-cycles and the multigrid's
masked levels, for the bounds-check build.

    python tests/bounds_cases_sweeps.py OUT.npz     (SG_LIBRARY_VARIANT=bounds selects that build)

Runs: the multi-sweep Jacobi tiles (a caller's scratch buffer takes them); Jacobi and SOR resident on
the chip with two, four and eight rows a thread; SOR to a tolerance with the checks in the launch,
native and mixed; Gauss-Seidel in one block, in chains of blocks and past 1024 cells a side; the
V-cycles with level launches, one-block tail and resident coarsest sweeps; one multigrid cycle, V and
W, around obstacles. Writes every result and the bounds-check record to OUT.npz."""
import importlib
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sg = importlib.import_module("python-game-engine_b200")
L = sg._lib

SHAPES = [(3, 65), (9, 33), (63, 77), (130, 67), (200, 151)]


def _masks(H, W):
    solid = np.zeros((H, W), bool)
    solid[[0, -1]] = solid[:, [0, -1]] = H > 4 and W > 4
    solid[H // 3:H // 2, W // 4:W // 2] = True
    return sg.operators.build_masks(torch.from_numpy(solid).cuda())


def cases():
    out = {}
    S = sg.solvers
    rng = np.random.default_rng(1)

    def run(name, H, W, dtype, solve, planes=True):
        p = torch.from_numpy(rng.uniform(-1, 1, (H, W))).to(dtype).cuda()
        div = torch.from_numpy(rng.uniform(-1, 1, (H, W))).to(dtype).cuda()
        fmu, fmv = _masks(H, W)[:2] if planes else (sg.RING_BOX, sg.RING_BOX)
        solve(p, div, fmu, fmv, 1.0, 1.0 / W, 0.5 / W)
        out[f"{name}_{H}x{W}_{'f32' if dtype == torch.float32 else 'f64'}"] = p.double().cpu().numpy()

    for dtype in (torch.float32, torch.float64):
        for H, W in SHAPES:
            scratch = torch.empty((H, W), dtype=dtype, device="cuda")
            run("jacobi_tiles", H, W, dtype, lambda *a: S.jacobi_pressure_solver(*a, iterations=11, scratch=scratch))
        for H, W in SHAPES + [(421, 300), (600, 801)]:
            run("jacobi", H, W, dtype, lambda *a: S.jacobi_pressure_solver(*a, iterations=21))
            run("sor", H, W, dtype, lambda *a: S.red_black_sor_gauss_seidel_pressure_solver(*a, iterations=9, omega=1.5),
                planes=False)
            run("tolerance", H, W, dtype, lambda *a: sg.SORToleranceSolver()(*a, tol=1e-30, max_iterations=17,
                                                                             check_every=5))
        for H, W, n in ((1, 7, 3), (63, 77, 9), (97, 161, 40), (33, 32, 75), (20, 1100, 2), (513, 520, 3),
                        (1030, 1027, 2)):
            run("gauss_seidel", H, W, dtype, lambda *a: S.gauss_seidel_pressure_solver(*a, iterations=n))
        for H, W, levels, smoother in ((64, 52, 3, "jacobi"), (136, 200, 4, "rb_sor_gauss_seidel"), (101, 130, 3, "jacobi"),
                                       (300, 260, 2, "rb_sor_gauss_seidel"), (63, 7, 1, "jacobi")):
            run("vcycles", H, W, dtype, lambda *a: sg.MultigridSolver()(*a, v_cycles=2, num_levels=levels,
                                                                        smoother_type=smoother, coarsest_iterations=6))
    for H, W in ((63, 77), (131, 203), (300, 421)):
        run("mixed_sor", H, W, torch.float32, lambda *a: sg.SORToleranceSolver()(
            *a, tol=1e-30, max_iterations=17, check_every=5, precision="mixed"))
        for prec in ("fp64", "fp32", "mixed"):
            for cycle in ("V", "W"):
                run(f"gmg_{prec}_{cycle}", H, W, torch.float32 if prec == "fp32" else torch.float64,
                    lambda *a: sg.GeometricMultigridSolver()(*a, precision=prec, fixed_cycles=1, cycle=cycle))
    torch.cuda.synchronize()
    line, unit = L.bounds_check()
    out["bounds_line"] = np.array(line)
    out["bounds_unit"] = np.array(unit)
    out["bounds_enabled"] = np.array(int(L.load().sg_bounds_check_enabled()))
    return out


if __name__ == "__main__":
    np.savez(sys.argv[1], **cases())
