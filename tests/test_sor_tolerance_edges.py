"""Sweeps to a tolerance from initial guesses so large that the first residual's sum of squares
overflows: the first chunk of sweeps is made all the same, whichever kernels make it."""
import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("CUDA device required", allow_module_level=True)

sg = package()


@pytest.mark.parametrize("shape,variant", [((40, 60), -1), ((40, 60), 0), ((40, 60), 1), ((600, 801), -1)])
def test_sweeps_start_from_an_overflowing_residual(shape, variant):
    H, W = shape
    p = torch.zeros((H, W), dtype=torch.float64, device="cuda")
    p[H // 2, W // 2] = 1e155  # residual 4e155, its square above the largest number; one sweep replaces it
    div = torch.rand((H, W), dtype=torch.float64, device="cuda")
    s = sg.SORToleranceSolver()
    s(p, div, sg.OPEN_BOX, sg.OPEN_BOX, 1.0, 1.0 / W, 0.5 / W, omega=1.0, tol=1e-6, max_iterations=100, check_every=50,
      variant=variant)
    assert s.last_iterations == 100 and not s.converged
    assert np.isfinite(s.last_relres) and bool(torch.isfinite(p).all())
