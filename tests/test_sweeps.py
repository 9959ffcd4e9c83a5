"""Sweeps with the iterate held on the chip (csrc/sweeps.cu) against the one-launch-per-sweep
kernels and the CPU oracle, bit for bit: grids at the edges of the blocks' regions (64 columns;
32, 64 or 128 rows), odd extents, every mask kind, row strides, sweep counts that end between
two trades of the blocks' frames, and the pipelined Gauss-Seidel wavefront in one and in
several passes, in one block and in a chain of blocks."""
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
L = sg._lib


def _case(H, W, npdt, kind, seed):
    rng = np.random.default_rng(seed)
    solid = np.zeros((H, W), bool)
    if kind == "planes":
        solid = O.box_solid(H, W)
        solid[H // 3:H // 3 + max(H // 6, 1), W // 4:W // 2] = True
    elif kind == "ring":
        solid = O.box_solid(H, W)
    fmu, fmv = O.face_masks_from_solid(solid)
    return (rng.uniform(-1, 1, (H, W)).astype(npdt), rng.uniform(-1, 1, (H, W)).astype(npdt), fmu, fmv)


def _mask_args(kind, fmu, fmv, W):
    if kind == "planes":
        t = [torch.from_numpy(x.astype(np.uint8)).cuda() for x in (fmu, fmv)]
        return t, (L.SG_MASK_PLANES, t[0].data_ptr(), W + 1, t[1].data_ptr(), W)
    return None, (L.SG_MASK_OPEN if kind == "open" else L.SG_MASK_RING, None, 0, None, 0)


@pytest.mark.parametrize("sor", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape,kind", [
    ((2, 2), "open"), ((5, 9), "ring"), ((32, 64), "open"), ((33, 65), "open"), ((17, 130), "planes"),
    ((49, 112), "planes"), ((50, 113), "open"), ((131, 67), "ring"), ((300, 310), "planes"), ((421, 300), "open"),
    ((600, 801), "planes"), ((1100, 90), "open")])
def test_resident_sweeps_equal_plain_kernels(sor, dtype, shape, kind):
    H, W = shape
    lib = L.load()
    s = L.stream_ptr()
    npdt = np.float32 if dtype == torch.float32 else np.float64
    p0, div, fmu, fmv = _case(H, W, npdt, kind, H + 3 * W)
    code = L.dtype_code(torch.empty((), dtype=dtype))
    keep, mask = _mask_args(kind, fmu, fmv, W)
    n = int(lib.sg_sweeps_workspace_bytes(code, H, W))
    assert n > 0
    ws = torch.full((n,), 1, dtype=torch.uint8, device="cuda")
    d = torch.zeros((H, W + 3), dtype=dtype, device="cuda")[:, :W]
    d.copy_(dev(div))
    for iters in (1, 2, 3, 4, 8, 9, 21):
        got = torch.zeros((H, W + 5), dtype=dtype, device="cuda")[:, :W]
        got.copy_(dev(p0))
        rc = lib.sg_sweeps_solve(code, sor, H, W, got.data_ptr(), W + 5, d.data_ptr(), W + 3, *mask, -0.37, 0.25, 1.9,
                                 iters, 0, ws.data_ptr(), n, s)
        assert rc == L.SG_OK, lib.sg_last_error()
        ref = dev(p0)
        if sor:
            rc = lib.sg_rbsor_solve(code, H, W, ref.data_ptr(), W, d.data_ptr(), W + 3, *mask, -0.37, 0.25, 1.9, iters, s)
        else:
            scratch = torch.empty_like(ref)
            rc = lib.sg_jacobi_solve(code, H, W, ref.data_ptr(), W, d.data_ptr(), W + 3, *mask, -0.37, 0.25, iters,
                                     scratch.data_ptr(), s)
        assert rc == L.SG_OK, lib.sg_last_error()
        torch.cuda.synchronize()
        assert torch.equal(got, ref), f"iterations {iters}: max {float((got - ref).abs().max()):.3e}"
    # from zero: p is not read
    got.fill_(float("nan"))
    ref.zero_()
    rc = lib.sg_sweeps_solve(code, sor, H, W, got.data_ptr(), W + 5, d.data_ptr(), W + 3, *mask, -0.37, 0.25, 1.9, 3, 1,
                             ws.data_ptr(), n, s)
    assert rc == L.SG_OK, lib.sg_last_error()
    rc = lib.sg_sweeps_solve(code, sor, H, W, ref.data_ptr(), W, d.data_ptr(), W + 3, *mask, -0.37, 0.25, 1.9, 3, 0,
                             ws.data_ptr(), n, s)
    assert rc == L.SG_OK, lib.sg_last_error()
    assert torch.equal(got, ref)


def test_resident_sweeps_refuse_what_does_not_fit():
    lib = L.load()
    p = torch.zeros((4000, 4000), device="cuda")
    assert lib.sg_sweeps_workspace_bytes(L.SG_F32, 4000, 4000) == 0
    rc = lib.sg_sweeps_solve(L.SG_F32, 1, 4000, 4000, p.data_ptr(), 4000, p.data_ptr(), 4000, L.SG_MASK_OPEN, None, 0,
                             None, 0, -1.0, 0.25, 1.5, 3, 0, p.data_ptr(), p.numel() * 4, L.stream_ptr())
    assert rc == L.SG_ERR_CAPACITY
    assert lib.sg_sweeps_workspace_bytes(7, 64, 64) == -1


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape,kind,iters", [((1, 7), "open", 3), ((2, 2), "open", 4), ((97, 161), "planes", 40),
                                              ((161, 97), "ring", 5), ((33, 32), "open", 75), ((180, 180), "open", 41),
                                              ((700, 260), "planes", 30), ((20, 1100), "planes", 2)])
def test_gauss_seidel_wave_equals_oracle(dtype, shape, kind, iters):
    H, W = shape
    p0, div, fmu, fmv = _case(H, W, dtype, kind, 7 * H + W)
    exp = p0.copy()
    O.gauss_seidel_pressure_solver(exp, div, fmu, fmv, 1.0, 1.0 / W, 0.5 / W, iterations=iters)
    got = dev(p0)
    mu, mv = (sg.OPEN_BOX,) * 2 if kind == "open" else ((sg.RING_BOX,) * 2 if kind == "ring" else (dev(fmu), dev(fmv)))
    sg.solvers.gauss_seidel_pressure_solver(got, dev(div), mu, mv, 1.0, 1.0 / W, 0.5 / W, iterations=iters)
    assert np.array_equal(got.cpu().numpy(), exp)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape,kind,iters", [
    ((2, 3), "open", 7), ((31, 33), "ring", 200), ((32, 900), "planes", 17), ((900, 32), "open", 64),
    ((513, 520), "planes", 3), ((600, 1024), "ring", 5), ((1024, 530), "open", 150)])
def test_gauss_seidel_chain_equals_one_block(dtype, shape, kind, iters):
    """Blocks with loaders of their own and without, rings that wrap, more sweeps than a launch holds."""
    H, W = shape
    lib = L.load()
    npdt = np.float32 if dtype == torch.float32 else np.float64
    p0, div, fmu, fmv = _case(H, W, npdt, kind, 11 * H + W)
    code = L.dtype_code(torch.empty((), dtype=dtype))
    keep, mask = _mask_args(kind, fmu, fmv, W)
    n = int(lib.sg_gauss_seidel_workspace_bytes(code, H, W, iters))
    ws = torch.full((max(n, 16),), 1, dtype=torch.uint8, device="cuda")
    got = torch.zeros((H, W + 5), dtype=dtype, device="cuda")[:, :W]
    got.copy_(dev(p0))
    ref, d = dev(p0), dev(div)
    args = (d.data_ptr(), W, *mask, -0.37, 0.25, iters)
    assert lib.sg_gauss_seidel_sweeps(code, H, W, got.data_ptr(), W + 5, *args, ws.data_ptr(), n, L.stream_ptr()) == 0
    assert lib.sg_gauss_seidel_solve(code, H, W, ref.data_ptr(), W, *args, L.stream_ptr()) == 0
    assert torch.equal(got, ref)
    if n:
        rc = lib.sg_gauss_seidel_sweeps(code, H, W, got.data_ptr(), W + 5, *args, ws.data_ptr(), n - 1, L.stream_ptr())
        assert rc == L.SG_ERR_ARG


@pytest.mark.parametrize("precision", ["native64", "native32", "mixed"])
@pytest.mark.parametrize("shape,kind,check,most", [((40, 60), "open", 7, 60), ((97, 161), "planes", 10, 95),
                                                   ((300, 310), "ring", 25, 400), ((1000, 901), "open", 3, 9)])
def test_sweeps_to_a_tolerance_equal_checked_launches(precision, shape, kind, check, most):
    """All checks in one launch against a launch per half sweep and a host check: the sweeps made, the iterate."""
    H, W = shape
    npdt = np.float64 if precision == "native64" else np.float32
    p0, div, fmu, fmv = _case(H, W, npdt, kind, 5 * H + W)
    mu, mv = (sg.OPEN_BOX,) * 2 if kind == "open" else ((sg.RING_BOX,) * 2 if kind == "ring" else (dev(fmu), dev(fmv)))
    out = []
    for variant in (-1, 0):
        for tol in (0.3, 1e-9):
            s = sg.solvers.SORToleranceSolver()
            p = dev(p0)
            s(p, dev(div), mu, mv, 1.0, 1.0 / W, 0.5 / W, omega=1.7, tol=tol, max_iterations=most, check_every=check,
              variant=variant, precision="mixed" if precision == "mixed" else "native")
            out.append((s.last_iterations, s.last_refinements, s.converged, s.last_relres, p))
    for a, b in zip(out[:2], out[2:]):
        assert a[:3] == b[:3]
        assert a[3] == pytest.approx(b[3], rel=1e-12)
        assert torch.equal(a[4], b[4])
