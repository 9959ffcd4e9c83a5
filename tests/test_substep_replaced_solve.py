"""A program that solves the pressure itself, by a solver of its own in the registry or by a
replaced step, may hand the simulation other tensors: the projection follows them."""
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("CUDA device required", allow_module_level=True)

sg = package()
FIELDS = ("density", "velocity_u", "velocity_v", "pressure", "divergence", "pressure_residual")


class CallByCall(sg.NullProfileSession):
    pass


def _sim(native):
    W, H = 52, 40
    cfg = sg.SimulationConfig(grid=sg.GridConfig(size=(W, H), cell_size=1.0 / W),
                              pressure_solver=sg.PressureSolverConfig(method="jacobi",
                                                                      params=sg.JacobiParams(iterations=20)))
    sim = sg.SmokeSimulation2D(cfg, None if native else CallByCall(), dtype=torch.float64, seed=5)
    sim.dt = 0.5 / W
    sim.add_plume(sg.PlumeSource(0.5 * W, 0.2 * H, 0.1 * H))
    return sim


@pytest.mark.parametrize("how", ["registry", "step"])
def test_projection_takes_the_pressure_of_the_programs_solve(how, monkeypatch):
    registry = __import__("importlib").import_module("python-game-engine_b200.registry")
    sims = [_sim(native) for native in (True, False)]
    for sim in sims:
        def solve(*args, sim=sim, **kwargs):
            sim.pressure = torch.cos(torch.arange(sim.pressure.numel(), device="cuda", dtype=torch.float64)
                                     ).reshape(sim.pressure.shape) * 1e-3
            sim.velocity_u = sim.velocity_u.clone()
        if how == "step":
            sim._solve_pressure = solve
        for step in range(3):
            if how == "registry":
                monkeypatch.setitem(registry.SOLVER_REGISTRY, ("jacobi", "cuda"), solve)
            sim.substep(sim.dt)
    for name in FIELDS:
        assert torch.equal(*(getattr(s, name) for s in sims)), name
