"""A substep's operators issued by two native calls against the same substep issued call by
call (which any profiler, subclass or replaced method still takes): every field bit for bit
over several steps, for every solver, both types and arithmetics, emitters with and without
heat, plumes, obstacles set on the way, and fields the program has replaced by strided ones."""
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("CUDA device required", allow_module_level=True)

sg = package()
simulation = __import__("importlib").import_module("python-game-engine_b200.simulation")
FIELDS = ("density", "velocity_u", "velocity_v", "pressure", "divergence", "pressure_residual", "_temperature")
PARAMS = {"jacobi": sg.JacobiParams(iterations=20), "gauss_seidel": sg.GaussSeidelParams(iterations=4),
          "rb_sor_gauss_seidel": sg.SORParams(iterations=10),
          "multigrid": sg.MultigridParams(smoother_type="rb_sor_gauss_seidel", num_levels=3),
          "rb_sor_tolerance": sg.SORToleranceParams(tol=1e-3, precision="native"),
          "geometric_multigrid": sg.GeometricMultigridParams(tol=1e-5, precision="mixed")}


class CallByCall(sg.NullProfileSession):
    pass


def _sim(method, dtype, W, H, heat, plume, arithmetic, native):
    cfg = sg.SimulationConfig(grid=sg.GridConfig(size=(W, H), cell_size=1.0 / W),
                              pressure_solver=sg.PressureSolverConfig(method=method, params=PARAMS[method]))
    sim = sg.SmokeSimulation2D(cfg, None if native else CallByCall(), dtype=dtype, seed=5)
    sim.dt = 0.5 / W
    sim.advection_arithmetic = sim.operator_arithmetic = arithmetic
    if heat is not None:
        sim.add_emitter(sg.Emitter2D((0.4 * W, 0.3 * H), 0.2 * H, 4.0, heat, (1.0, 3.0), approach="quadratic"))
        sim.add_emitter(sg.Emitter2D((0.7 * W, 0.5 * H), 0.1 * H, 2.0, 0.0, (0.0, -3.0), approach="gaussian"))
    if plume:
        sim.add_plume(sg.PlumeSource(0.5 * W, 0.2 * H, 0.1 * H, noise_amp=0.05))
    return sim


@pytest.mark.parametrize("method", sorted(PARAMS))
@pytest.mark.parametrize("dtype,heat,plume,arithmetic", [
    (torch.float32, 12.0, False, "reference"), (torch.float64, None, True, "reference"),
    (torch.float32, 0.0, True, "float32"), (torch.float32, 6.0, True, "float32")])
def test_native_substep_equals_call_by_call(method, dtype, heat, plume, arithmetic, monkeypatch):
    W, H = 52, 40
    sims = [_sim(method, dtype, W, H, heat, plume, arithmetic, native) for native in (True, False)]
    taken = []
    run = simulation.SmokeSimulation2D._native_substep
    monkeypatch.setattr(simulation.SmokeSimulation2D, "_native_substep", lambda s, p: taken.append(s) or run(s, p))
    for step in range(5):
        if step == 2:
            solid = torch.zeros((H, W), dtype=torch.bool)
            solid[[0, -1]] = solid[:, [0, -1]] = True
            solid[18:23, 20:30] = True
            for s in sims:
                s.set_solid_mask(solid)
        if step == 3:  # a field of the program's own, wider rows
            for s in sims:
                wide = torch.zeros((H, W + 6), dtype=dtype, device="cuda")[:, :W]
                wide.copy_(s.density)
                s.density = wide
        for s in sims:
            s.update(s.dt) if heat is not None else s.substep(s.dt)
        for name in FIELDS:
            a, b = (getattr(s, name) for s in sims)
            assert torch.equal(a, b), (step, name)
    assert len(taken) == 5 and all(s is sims[0] for s in taken)
    assert sims[0].step_index == sims[1].step_index == 5


def test_replaced_steps_and_fields_are_honoured(monkeypatch):
    sim = _sim("jacobi", torch.float32, 40, 32, 5.0, False, "reference", True)
    calls = []
    monkeypatch.setattr(simulation.SmokeSimulation2D, "_native_substep", lambda *a: calls.append("native"))
    sim._apply_forces = lambda dt: calls.append("forces")
    sim.substep(sim.dt)
    assert calls == ["forces"]
    del sim._apply_forces
    sim.density = sim.density.double()
    with pytest.raises(TypeError):
        sim.substep(sim.dt)
    assert calls == ["forces"]
