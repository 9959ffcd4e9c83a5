"""The fused reference V-cycles from p = 0, which do not read the pressure, against the separate
kernels on a cleared one, bit for bit: level launches, one-block tail, one level resident on the
chip, no coarsest sweeps, row strides, a pressure that holds NaN."""
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


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("smoother", ["jacobi", "rb_sor_gauss_seidel"])
@pytest.mark.parametrize("shape,levels,nu,nu_c", [
    ((48, 40), 3, 2, 9), ((48, 40), 1, 2, 9), ((136, 200), 4, 2, 30), ((136, 200), 2, 1, 0), ((101, 130), 3, 2, 25),
    ((101, 130), 1, 2, 0)])
def test_cycles_from_zero(dtype, smoother, shape, levels, nu, nu_c, monkeypatch):
    H, W = shape
    rng = np.random.default_rng(H * W + levels)
    solid = O.box_solid(H, W)
    solid[H // 3:H // 2, W // 4:W // 2] = True
    fmu, fmv = (dev(x) for x in O.face_masks_from_solid(solid))
    div = dev(rng.uniform(-1, 1, (H, W)).astype(dtype))
    kw = dict(v_cycles=2, smoother_type=smoother, num_levels=levels, smoother_iterations=nu, coarsest_iterations=nu_c)
    wide = torch.full((H, W + 7), float("nan"), dtype=div.dtype, device="cuda")
    seen = []
    fused = sg.MultigridSolver._fused
    monkeypatch.setattr(sg.MultigridSolver, "_fused", lambda *a: seen.append(fused(*a)) or seen[-1])
    sg.MultigridSolver()(wide[:, :W], div, fmu, fmv, 1.0, 1.0 / W, 0.5 / W, zero_initial_guess=True, **kw)
    assert seen == [True] and bool(torch.isnan(wide[:, W:]).all())
    monkeypatch.setattr(sg.MultigridSolver, "_fused", lambda *a: False)
    ref = torch.zeros((H, W), dtype=div.dtype, device="cuda")
    sg.MultigridSolver()(ref, div, fmu, fmv, 1.0, 1.0 / W, 0.5 / W, **kw)
    assert torch.equal(wide[:, :W], ref)
