"""Sweeps with the iterate held on the chip where the other tests do not reach: more sweeps than one
launch makes, and sweeps to a tolerance with eight rows a thread (checked from the host), against
the one-launch-per-sweep kernels bit for bit."""
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("CUDA device required", allow_module_level=True)

sg = package()
L = sg._lib


@pytest.mark.parametrize("sor", [0, 1])
def test_more_sweeps_than_a_launch_makes(sor):
    H, W, n = 66, 70, 16384 + 37
    p = torch.rand((H, W), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    d = p.flip(0) - p.mean()
    ref = p.clone()
    mask = (L.SG_MASK_OPEN, None, 0, None, 0)
    nbytes = int(L.load().sg_sweeps_workspace_bytes(L.SG_F64, H, W))
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    args = (d.data_ptr(), W, *mask, -0.37, 0.25)
    L.call("sg_sweeps_solve", L.SG_F64, sor, H, W, p.data_ptr(), W, *args, 1.3, n, 0, ws.data_ptr(), nbytes,
           L.stream_ptr())
    if sor:
        L.call("sg_rbsor_solve", L.SG_F64, H, W, ref.data_ptr(), W, *args, 1.3, n, L.stream_ptr())
    else:
        scratch = torch.empty_like(ref)
        L.call("sg_jacobi_solve", L.SG_F64, H, W, ref.data_ptr(), W, *args, n, scratch.data_ptr(), L.stream_ptr())
    assert torch.equal(p, ref)


@pytest.mark.parametrize("precision", ["native64", "native32", "mixed"])
@pytest.mark.parametrize("shape", [(600, 801), (800, 900)])
def test_tolerance_with_eight_rows_a_thread(precision, shape):
    H, W = shape
    dtype = torch.float64 if precision == "native64" else torch.float32
    g = torch.Generator("cuda").manual_seed(H)
    p0, div = (torch.rand((H, W), dtype=dtype, device="cuda", generator=g) - 0.5 for _ in range(2))
    assert L.load().sg_sweeps_workspace_bytes(L.dtype_code(p0), H, W) > 0
    out = []
    for variant in (-1, 0):
        s = sg.SORToleranceSolver()
        p = p0.clone()
        s(p, div, sg.OPEN_BOX, sg.OPEN_BOX, 1.0, 1.0 / W, 0.5 / W, omega=1.7, tol=1e-9, max_iterations=70, check_every=8,
          variant=variant, precision="mixed" if precision == "mixed" else "native")
        out.append((s.last_iterations, s.last_refinements, s.last_relres, p))
    assert out[0][:3] == out[1][:3]
    assert torch.equal(out[0][3], out[1][3])
