"""Kernels are placed while their predecessor in the stream drains (physica_b200/csrc/dependent_launch.cuh) and
must still see everything the stream ran before them: steps enqueued back to back, their inputs written
and their outputs read by other kernels of the stream, give the bits of steps with a synchronisation
around each.  And every kind of step gives the bits of a process that waits for each kernel."""
import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest
import torch

if __name__ == "__main__":
    sys.path.insert(0, str(pathlib.Path(__file__).resolve().parents[1]))

from physica_b200 import pbf, scenes, sph

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


def every_kind():
    """Outputs of a few steps of each kind, enqueued without waiting."""
    out = {}

    def steps(name, solver, state, control, params, cache, count=4):
        following = solver.allocate_state()
        for k in range(count):
            control.external_accelerations.mul_(1.01).add_(0.1 * k)
            solver.forward_step(state, control, params, following, cache)
            out[f"{name}{k}"] = following.positions * 2.0 + following.velocities
            state, following = following, state
        return following, state   # the last step's input and output

    def adjoint(name, solver, state, control, params, following, cache, kind):
        seed = following.positions.double() + following.velocities.double()
        na, pa = solver.allocate_state_adjoint(), solver.allocate_state_adjoint()
        na.positions.copy_(seed)
        na.velocities.copy_(seed - 1.0)
        ca, qa = solver.allocate_control_adjoint(), solver.allocate_parameter_adjoint()
        solver.vjp_step(state, control, params, following, cache, na, pa, ca, qa)
        out[name + "_adjoint"] = pa.positions + pa.velocities
        out[name + "_masses"] = qa.tensors["masses"].clone()
        if kind == "pbf":
            tangent = solver.allocate_state_tangent()
            solver.jvp_step(state, control, params, following, cache, pbf.StateTangent(following.velocities * 0.01, following.positions),
                            control, solver.allocate_parameter_tangent(), tangent)
            out[name + "_tangent"] = tangent.positions + tangent.velocities

    scene = lambda n, **o: scenes.dam_break((n, n, n), (0.0, 0.0, 0.0), (2.0 * n * 0.0125 + 0.05,) * 3, 3, 3, velocity_sigma=0.4, **o)
    for n in (16, 30, 57):
        made = pbf.solver_for_scene(scene(n))
        steps(f"forward{n}_", *made, made[0].allocate_step_cache())
    made = pbf.solver_for_scene(scenes.with_boundary(scene(20), 4))
    steps("boundary", *made, made[0].allocate_step_cache())
    for recompute in (False, True):
        made = pbf.solver_for_scene(scene(24), mode=pbf.ExecutionMode.differentiable)
        made[0].set_checkpoint_recompute(recompute)
        cache = made[0].allocate_step_cache()
        last, following = steps(f"gradient{recompute}", *made, cache, count=2)
        adjoint(f"gradient{recompute}", made[0], last, made[2], made[3], following, cache, "pbf")
    batch, state, control, params = pbf.batch_for_scenes([scenes.batched_scene(c, 200 + k, 3) for k, c in enumerate((1500, 4000, 257))])
    steps("batch", batch, state, control, params, 0)
    for method in sph.Method:
        s = scene(24, dt=scenes.SPH_DT)
        s.sph = scenes.sph_parameter_arrays(s, method=method.name)
        made = sph.solver_for_scene(s, method, mode=pbf.ExecutionMode.differentiable)
        cache = made[0].allocate_step_cache()
        last, following = steps(method.name, *made, cache, count=3)
        adjoint(method.name, made[0], last, made[2], made[3], following, cache, "sph")
    torch.cuda.synchronize()
    return {k: t.cpu().numpy() for k, t in out.items()}


def test_every_kind_of_step_equals_one_that_waits_for_each_kernel(tmp_path):
    path = tmp_path / "waited.npz"
    subprocess.run([sys.executable, __file__, str(path)], check=True, env={**os.environ, "CUDA_LAUNCH_BLOCKING": "1"}, timeout=600)
    waited, enqueued = np.load(path), every_kind()
    assert sorted(waited.files) == sorted(enqueued)
    for name, value in enqueued.items():
        np.testing.assert_array_equal(value, waited[name], err_msg=name)


if __name__ == "__main__":
    np.savez(sys.argv[1], **every_kind())
