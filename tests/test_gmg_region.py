"""The multigrid's region kernels (csrc/gmg_region.cuh) against the oracle's cycle: grids around
the regions' sizes (32 x 64 cells, 64-cell tail), odd extents, obstacles down to the coarsest
level, one-cell walls, W-cycles, one to three sweeps a side, a fine level with a closed face
between fluid cells (grid-wide kernels there), and solves that start from a given pressure.
Tolerances: one cycle 1e-10 relative in float64, 2e-5 with float32 cycles (rounding of a few
hundred dependent operations, as for the other level kernels)."""
import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("CUDA device required", allow_module_level=True)

import oracle as O  # noqa: E402
from cuda_adapter import dev  # noqa: E402

sg = package()


def _problem(H, W, obstacles, seed):
    rng = np.random.default_rng(seed)
    solid = np.zeros((H, W), bool)
    if obstacles:
        solid = O.box_solid(H, W)
        solid[H // 3:H // 3 + max(H // 5, 1), W // 4:W // 2] = True
        solid[3 * H // 4, : W // 3] = True
    fmu, fmv = O.face_masks_from_solid(solid)
    fl = O.is_fluid_from_faces(fmu, fmv)
    div = rng.standard_normal((H, W)) * fl
    div -= fl * (div.sum() / fl.sum())
    return fmu, fmv, fl, div


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("shape,cycle,sweeps,obstacles", [
    ((64, 64), "V", (2, 2), False), ((65, 66), "V", (2, 2), True), ((33, 130), "W", (2, 1), True),
    ((150, 95), "V", (3, 3), True), ((129, 257), "V", (1, 1), False), ((63, 17), "W", (2, 2), True),
    ((300, 421), "V", (2, 2), True), ((40, 52), "V", (0, 2), True)])
def test_cycle_matches_oracle(precision, shape, cycle, sweeps, obstacles):
    H, W = shape
    fmu, fmv, fl, div = _problem(H, W, obstacles, H + W)
    gmg = O.GMGOracle(fmu, fmv, fl, coarsest=8, omega=1.3, pre=sweeps[0], post=sweeps[1], cycle=cycle)
    exp = np.zeros((H, W))
    gmg.vcycle(0, exp, -0.7 * div)
    p = torch.zeros((H, W), dtype=torch.float32 if precision == "fp32" else torch.float64, device="cuda")
    solver = sg.GeometricMultigridSolver()
    solver(p, dev(div.astype(np.float32) if precision == "fp32" else div), dev(fmu), dev(fmv), 0.7, 1.0, 1.0,
           precision=precision, fixed_cycles=1, coarsest=8, cycle=cycle, pre_sweeps=sweeps[0], post_sweeps=sweeps[1])
    got = p.double().cpu().numpy()
    tol = 1e-10 if precision == "fp64" else 2e-5
    assert np.max(np.abs(got - exp)) <= tol * np.max(np.abs(exp))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("closed_face", [False, True])
def test_reported_residual_around_obstacles_is_true(precision, closed_face):
    """The carried residual r - A e is the true one of the returned pressure, from a zero guess
    and from a given pressure, also when a face between two fluid cells is closed. (One-cell walls
    vanish from the coarse levels, so these solves slow down far above 1e-8; what they report
    has to be true all the same.)"""
    H, W = 131, 203
    fmu, fmv, fl, div = _problem(H, W, True, 5)
    if closed_face:
        fmu[H // 5, W // 7] = False
        div = div * O.is_fluid_from_faces(fmu, fmv)
    h, dt = 1.0 / W, 0.5 / W
    alpha = O.alpha_coeff(h, 1.0, dt)
    for start in (None, 7):
        p0 = np.zeros((H, W)) if start is None else np.random.default_rng(start).standard_normal((H, W)) * fl
        p = dev(p0)
        solver = sg.GeometricMultigridSolver()
        solver(p, dev(div), dev(fmu), dev(fmv), 1.0, h, dt, precision=precision, tol=1e-8, max_cycles=80,
               zero_initial_guess=start is None)
        r = O.compute_residual(p.cpu().numpy(), div, fl, fmu, fmv, alpha, 0.25, np.empty((H, W)))
        rel = np.linalg.norm(r) / np.linalg.norm(alpha * div * fl)
        assert abs(rel - solver.last_relres) <= 1e-3 * max(solver.last_relres, 1e-8) + 1e-11
