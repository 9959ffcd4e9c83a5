"""What a tolerance solve of the convergent multigrid reports near the rounding floor, on grids whose
fine level runs the region kernels or the one-block tail: the relative residual is that of the
returned pressure, not of a recurrence that goes on falling where the pressure no longer changes.

The divergence is the lowest cosine mode, so that the pressure exceeds the right-hand side by some
(W / pi)^2 and its own rounding leaves a residual of 1e-13 to 1e-12. Forming the residual from
differences of neighbours costs a few roundings of |grad p| <= W / 3 of the right-hand side, some
1e-14: a tenth of the floor covers the two evaluations' difference."""
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


def _true_relres(p, b, fmu, fmv):
    p, r = p.astype(np.longdouble), b.astype(np.longdouble)
    x = (p[:, 1:] - p[:, :-1]) * fmu[:, 1:-1]
    r[:, :-1] += x
    r[:, 1:] -= x
    y = (p[1:] - p[:-1]) * fmv[1:-1]
    r[:-1] += y
    r[1:] -= y
    return float(np.sqrt((r ** 2).sum() / (b.astype(np.longdouble) ** 2).sum()))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,obstacle", [((200, 256), False), ((131, 203), True), ((300, 421), True),
                                            ((60, 64), True)])
def test_reported_residual_at_the_rounding_floor(precision, shape, obstacle):
    H, W = shape
    solid = np.zeros((H, W), bool)
    if obstacle:
        solid[H // 3:H // 2, W // 4:W // 2] = True
    fmu, fmv = O.face_masks_from_solid(solid)
    fl = O.is_fluid_from_faces(fmu, fmv)
    div = np.cos(np.pi * (np.arange(W) + 0.5) / W)[None, :] * np.ones((H, 1)) * fl
    div -= fl * (div.sum() / fl.sum())
    h, dt = 1.0 / W, 0.5 / W
    b = O.alpha_coeff(h, 1.0, dt) * div
    p = torch.zeros((H, W), dtype=torch.float64, device="cuda")
    solver = sg.GeometricMultigridSolver()
    solver(p, dev(div), dev(fmu), dev(fmv), 1.0, h, dt, precision=precision, tol=1e-15, max_cycles=40,
           zero_initial_guess=True)
    true = _true_relres(p.cpu().numpy(), b, fmu, fmv)
    assert not solver.converged and true > 1e-15
    assert abs(solver.last_relres - true) <= 0.1 * true + 2e-14
