"""Kernels are placed while their predecessor in the stream drains (physica_b200/csrc/dependent_launch.cuh) and
must still see everything the stream ran before them: steps enqueued back to back, their inputs written
and their outputs read by other kernels of the stream, give the bits of steps with a synchronisation
around each."""
import numpy as np
import pytest
import torch

from physica_b200 import pbf, scenes

pytestmark = pytest.mark.gpu


def chain(count, mode, synchronise, graph):
    n = int(round(count ** (1 / 3)))
    scene = scenes.dam_break((n, n, n), (0.0, 0.0, 0.0), (2.0 * n * 0.0125 + 0.05,) * 3, 3, 3, velocity_sigma=0.4)
    differentiable = mode == "gradient"
    solver, state, control, params = pbf.solver_for_scene(
        scene, mode=pbf.ExecutionMode.differentiable if differentiable else pbf.ExecutionMode.forward)
    if graph:
        solver.set_graph_mode(True)
    cache, following = solver.allocate_step_cache(), solver.allocate_state()
    wait = torch.cuda.synchronize if synchronise else (lambda: None)
    out = []
    for k in range(6):
        control.external_accelerations.mul_(1.01).add_(0.1 * k)   # inputs written just before
        wait()
        solver.forward_step(state, control, params, following, cache)
        wait()
        out.append(following.positions * 2.0 + following.velocities)   # outputs read just after
        if differentiable:
            adjoint = pbf.StateAdjoint(out[-1].double(), out[-1].double() - 1.0)
            pa, ca, qa = solver.allocate_state_adjoint(), solver.allocate_control_adjoint(), solver.allocate_parameter_adjoint()
            wait()
            solver.vjp_step(state, control, params, following, cache, adjoint, pa, ca, qa)
            wait()
            out += [pa.positions + pa.velocities, ca.external_accelerations.clone()]
        state, following = following, state
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in out]


@pytest.mark.parametrize("count", [512, 27000, 216000])
@pytest.mark.parametrize("mode,graph", [("forward", False), ("forward", True), ("gradient", False)])
def test_steps_enqueued_back_to_back(count, mode, graph):
    for a, b in zip(chain(count, mode, True, False), chain(count, mode, False, graph)):
        np.testing.assert_array_equal(a, b)
