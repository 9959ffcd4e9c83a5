"""The reference's V-cycles in two launches per level (csrc/vcycle.cu) against the same cycles
built from the separate kernels, bit for bit: grids around the tiles' sizes (64 columns; 32 and
64 rows), hierarchies that end in and above the one-block tail, one level only, no smoothing,
the most sweeps a side that the tiles take, masks with obstacles, row strides."""
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
@pytest.mark.parametrize("shape,levels,nu,nu_c,obstacles", [
    ((64, 64), 4, 2, 30, False), ((66, 64), 2, 2, 9, True), ((128, 192), 6, 2, 30, True), ((136, 120), 4, 4, 7, True),
    ((300, 260), 2, 1, 41, True), ((48, 1040), 5, 3, 30, False), ((50, 75), 3, 2, 12, True), ((96, 96), 3, 0, 0, False),
    ((1024, 1088), 7, 2, 30, True)])
def test_fused_cycles_equal_separate_kernels(dtype, smoother, shape, levels, nu, nu_c, obstacles, monkeypatch):
    H, W = shape
    rng = np.random.default_rng(H + W + levels)
    solid = np.zeros((H, W), bool)
    if obstacles:
        solid = O.box_solid(H, W)
        solid[H // 3:H // 3 + max(H // 8, 1), W // 4:W // 2] = True
    fmu, fmv = (dev(x) for x in O.face_masks_from_solid(solid))
    p0 = dev(rng.uniform(-1, 1, (H, W)).astype(dtype))
    div = dev(rng.uniform(-1, 1, (H, W)).astype(dtype))
    solver = sg.MultigridSolver()

    def run(p):
        solver(p, div, fmu, fmv, 1.0, 1.0 / W, 0.5 / W, v_cycles=2, smoother_type=smoother, num_levels=levels,
               smoother_iterations=nu, coarsest_iterations=nu_c)
        torch.cuda.synchronize()
        return p

    got = torch.full((H, W + 7), 3.0, dtype=p0.dtype, device="cuda")
    got[:, :W] = p0
    seen = []
    fused = sg.MultigridSolver._fused
    monkeypatch.setattr(sg.MultigridSolver, "_fused", lambda *a: seen.append(fused(*a)) or seen[-1])
    run(got[:, :W])
    assert seen == [True]
    monkeypatch.setattr(sg.MultigridSolver, "_fused", lambda *a: False)
    ref = run(p0.clone())
    assert torch.equal(got[:, :W], ref), f"max {float((got[:, :W] - ref).abs().max()):.3e}"
    assert bool((got[:, W:] == 3.0).all())


def test_other_smoothers_and_counts_keep_the_separate_kernels():
    H = W = 64
    solver = sg.MultigridSolver()
    p, div = torch.zeros((H, W), device="cuda"), torch.randn((H, W), device="cuda")
    kw = dict(v_cycles=1, num_levels=3, coarsest_iterations=5)
    solver(p, div, sg.OPEN_BOX, sg.OPEN_BOX, 1.0, 1.0 / W, 0.5 / W, smoother_type="gauss_seidel", **kw)
    solver(p, div, sg.OPEN_BOX, sg.OPEN_BOX, 1.0, 1.0 / W, 0.5 / W, smoother_type="jacobi", smoother_iterations=9, **kw)
    solver(p, div.double(), sg.OPEN_BOX, sg.OPEN_BOX, 1.0, 1.0 / W, 0.5 / W, **kw)
    assert solver._workspace is None and bool(torch.isfinite(p).all())
