"""Solves whose block 1 gives up its waits for other blocks, for the bounds-check build.

    SG_LIBRARY_VARIANT=bounds python tests/lost_waits.py OUT.npz

Each case is run three times: as it is, with block 1's waits given up, and as it is again. Writes
the three pressures, the lost waits counted and what the call raised."""
import importlib
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sg = importlib.import_module("python-game-engine_b200")
L = sg._lib


def solves():
    """name -> a call on (pressure, divergence, mask u, mask v, density, cell size, dt)."""
    S = sg.solvers
    return {
        "jacobi": lambda *a: S.jacobi_pressure_solver(*a, iterations=90),
        "sor": lambda *a: S.red_black_sor_gauss_seidel_pressure_solver(*a, iterations=41, omega=1.5),
        # 4 sweeps: the last trade is the first one that block 1 gives up
        "sor_one_trade": lambda *a: S.red_black_sor_gauss_seidel_pressure_solver(*a, iterations=4, omega=1.5),
        "gauss_seidel": lambda *a: S.gauss_seidel_pressure_solver(*a, iterations=40),
        "vcycles": lambda *a: sg.MultigridSolver()(*a, v_cycles=1, num_levels=1, coarsest_iterations=30),
        "tolerance": lambda *a: sg.SORToleranceSolver()(*a, omega=1.5, tol=0.4, max_iterations=400, check_every=4),
        "mixed": lambda *a: sg.SORToleranceSolver()(*a, omega=1.5, tol=0.4, max_iterations=400, check_every=4,
                                                    precision="mixed"),
    }


def main(out_path):
    out = {}
    H, W = 200, 150
    rng = np.random.default_rng(3)
    div = torch.from_numpy(rng.uniform(-1, 1, (H, W)).astype(np.float32)).cuda()
    for name, solve in solves().items():
        for run, block in (("before", -1), ("lost", 1), ("after", -1)):
            L.check(L.load().sg_bounds_lose_waits(block), "sg_bounds_lose_waits")
            p = torch.zeros((H, W), device="cuda")
            raised = ""
            try:
                solve(p, div, sg.OPEN_BOX, sg.OPEN_BOX, 1.0, 1.0 / W, 0.5 / W)
            except L.SmokeCudaError as e:
                raised = str(e)
            out[f"{name}_{run}"] = p.cpu().numpy()
            out[f"{name}_{run}_count"] = np.array(L.lost_waits())
            out[f"{name}_{run}_raised"] = np.array(raised)
    np.savez(out_path, **out)


if __name__ == "__main__":
    main(sys.argv[1])
