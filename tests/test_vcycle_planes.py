"""The reference's V-cycles on the caller's own mask planes and fields, fused against the separate
kernels: planes that are views into wider rows, planes that a program edits between calls, planes
that no kernel can read, fields that share memory or are expanded, counts below one."""
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


def _problem(H, W, dtype=np.float32):
    rng = np.random.default_rng(3 * H + W)
    solid = O.box_solid(H, W)
    solid[H // 3:H // 3 + max(H // 6, 1), W // 4:W // 2] = True
    fmu, fmv = (dev(x) for x in O.face_masks_from_solid(solid))
    return fmu, fmv, dev(rng.uniform(-1, 1, (H, W)).astype(dtype)), dev(rng.uniform(-1, 1, (H, W)).astype(dtype))


def _run(solver, p, div, fmu, fmv, **kw):
    H, W = p.shape
    args = dict(v_cycles=2, num_levels=3, smoother_type="rb_sor_gauss_seidel", coarsest_iterations=6)
    args.update(kw)
    solver(p, div, fmu, fmv, 1.0, 1.0 / W, 0.5 / W, **args)
    return p


def _wide(m):
    """The same plane as a view into rows that are five bytes longer, all faces open there."""
    w = torch.ones((m.shape[0], m.shape[1] + 5), dtype=m.dtype, device=m.device)
    w[:, :m.shape[1]] = m
    return w[:, :m.shape[1]]


@pytest.mark.parametrize("shape", [(48, 40), (136, 200)])
@pytest.mark.parametrize("smoother", ["jacobi", "rb_sor_gauss_seidel"])
@pytest.mark.parametrize("levels", [1, 3])
def test_planes_in_wider_rows(shape, smoother, levels):
    fmu, fmv, p0, div = _problem(*shape)
    kw = dict(smoother_type=smoother, num_levels=levels)
    exp = _run(sg.MultigridSolver(), p0.clone(), div, fmu, fmv, **kw)
    got = _run(sg.MultigridSolver(), p0.clone(), div, _wide(fmu), _wide(fmv), **kw)
    assert torch.equal(got, exp)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(48, 40), (136, 200), (51, 33)])
def test_planes_edited_between_calls(shape, dtype, monkeypatch):
    """Without rebuild_masks the coarser levels and the cells stay those of the first call; the fine
    level's faces are the planes' as they are."""
    H, W = shape
    fmu, fmv, p0, div = _problem(H, W, dtype)
    fused = sg.MultigridSolver._fused
    out = []
    for f in (fused, lambda *a: False):
        monkeypatch.setattr(sg.MultigridSolver, "_fused", f)
        mu, mv = fmu.clone(), fmv.clone()
        solver = sg.MultigridSolver()
        first = _run(solver, p0.clone(), div, mu, mv)
        mu[H // 2 + 2:H - 3, W // 2 + 3] = False               # a wall inside
        mu[4, 5:8] = mv[4:6, 5:7] = False                      # cells that lose all their faces
        mv[H // 3 + 1, W // 4:W // 2] = mu[H // 3, W // 4:W // 2] = True  # and gain some
        out.append((first, _run(solver, p0.clone(), div, mu, mv)))
    assert torch.equal(out[0][0], out[1][0])
    assert not torch.equal(out[0][0], out[0][1])
    assert torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("bad", ["taller", "wider", "int32", "transposed", "host", "u for v"])
def test_planes_that_cannot_be_read_are_refused(bad):
    H, W = 48, 40
    fmu, fmv, p, div = _problem(H, W)
    if bad == "taller":
        fmu, fmv = (torch.cat([m, m[:8]]).contiguous() for m in (fmu, fmv))
    elif bad == "wider":
        fmu, fmv = (torch.cat([m, m[:, :8]], 1).contiguous() for m in (fmu, fmv))
    elif bad == "int32":
        fmu, fmv = fmu.int(), fmv.int()
    elif bad == "transposed":
        fmu, fmv = (m.t().contiguous().t() for m in (fmu, fmv))
    elif bad == "host":
        fmu, fmv = fmu.cpu(), fmv.cpu()
    else:
        fmv = fmu
    before = p.clone()
    solver = sg.MultigridSolver()
    for _ in range(2):
        with pytest.raises((ValueError, TypeError)):
            _run(solver, p, div, fmu, fmv)
    assert torch.equal(p, before)


@pytest.mark.parametrize("shape", [(48, 40), (136, 200)])
def test_fields_that_share_memory(shape):
    H, W = shape
    fmu, fmv, p0, div = _problem(H, W)
    exp = _run(sg.MultigridSolver(), p0.clone(), div[:1].expand(H, W).contiguous(), fmu, fmv)
    assert torch.equal(_run(sg.MultigridSolver(), p0.clone(), div[:1].expand(H, W), fmu, fmv), exp)
    exp = _run(sg.MultigridSolver(), p0.clone(), p0.clone(), fmu, fmv)
    both = p0.clone()
    assert torch.equal(_run(sg.MultigridSolver(), both, both, fmu, fmv), exp)


@pytest.mark.parametrize("cycles", [0, -1])
def test_no_cycles(cycles):
    fmu, fmv, p0, div = _problem(48, 40)
    assert torch.equal(_run(sg.MultigridSolver(), p0.clone(), div, fmu, fmv, v_cycles=cycles), p0)
    p = _run(sg.MultigridSolver(), p0.clone(), div, fmu, fmv, v_cycles=cycles, zero_initial_guess=True)
    assert not bool(p.any())
