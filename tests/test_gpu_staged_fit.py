"""Which passes a step takes follows how dense its particles are (physica_b200/csrc/staged_fit.h): lattices whose
stencil columns outgrow the staged passes' records run the per-lane passes from the step after the first measurement on,
and every step has the bits of the per-lane solver.  The routes differ by one kernel launch."""

import numpy as np
import pytest
import torch

from physica_b200 import pbf, scenes, sph

pytestmark = pytest.mark.gpu

ITERATIONS = 2
PBF_LAUNCHES = {True: 9 + 2 * ITERATIONS, False: 10 + 2 * ITERATIONS}   # by staged


def lattice(count, ratio, h=0.025, **options):
    """A jittered block of about `count` particles, `ratio` of them to a support radius."""
    n = int(round(count ** (1 / 3)))
    spacing = h / ratio
    s = scenes.dam_break((n, n, n), (0.0, 0.0, 0.0), (2.0 * (n + 3) * spacing,) * 3, 5, ITERATIONS, h=h, velocity_sigma=0.1, **options)
    at = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij")).reshape(3, -1)
    jitter = 0.1 * (2.0 * np.random.default_rng(6).random(at.shape) - 1.0)
    s.positions[:] = ((at + 1 + jitter) * spacing).astype(np.float32)
    s.masses[:] = np.float32(1000.0 * spacing ** 3)
    return s


def steps(solver, state, control, params, count):
    """The outputs and the kernel launches of `count` steps, each waited for."""
    cache, following = solver.allocate_step_cache(), solver.allocate_state()
    out, launches = [], []
    for _ in range(count):
        before = pbf.launch_count()
        solver.forward_step(state, control, params, following, cache)
        launches.append(pbf.launch_count() - before)
        torch.cuda.synchronize()
        out += [following.positions.cpu().numpy(), following.velocities.cpu().numpy()]
        state, following = following, state
    return out, launches


def run(scene, shape, count=3, graph=False):
    solver, state, control, params = pbf.solver_for_scene(scene)
    solver.launch_shape = shape
    solver.set_graph_mode(graph)
    return steps(solver, state, control, params, count)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("count,ratio,staged", [(8000, 2.0, True), (8000, 2.4, False), (8000, 3.0, True),
                                                (64000, 2.0, False), (64000, 2.9, False), (64000, 4.0, False),
                                                (185193, 2.0, True), (185193, 2.3, False), (185193, 3.2, False)])
def test_density_decides(count, ratio, staged, graph):
    """At a radius of 2.8 spacings and more lists of slots overflow: a small scene stays with the staged passes and their hit
    masks, the others keep hit masks in the per-lane passes."""
    scene = lattice(count, ratio)
    out, launches = run(scene, pbf.LaunchShape(4, 128, 128), graph=graph)
    assert launches[1:] == [PBF_LAUNCHES[staged]] * 2, launches
    for a, b in zip(out, run(scene, pbf.LaunchShape(0, 128, 128))[0]):
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32))


def test_new_inputs_are_measured_again():
    """A solver that is handed a dense state after a loose one, and back, follows within its 16 steps."""
    scene = lattice(8000, 2.0)
    dense = torch.from_numpy(lattice(8000, 2.4).positions).cuda()
    solver, state, control, params = pbf.solver_for_scene(scene)
    loose, cache, following = state.positions.clone(), solver.allocate_step_cache(), solver.allocate_state()
    for positions, staged in ((loose, True), (dense, False), (loose, True)):
        state.positions.copy_(positions)
        for _ in range(18):
            solver.forward_step(state, control, params, following, cache)
            torch.cuda.synchronize()
            state.step_index += 1
        counts = []
        for _ in range(2):
            before = pbf.launch_count()
            solver.forward_step(state, control, params, following, cache)
            state.step_index += 1
            counts.append(pbf.launch_count() - before)
        assert min(counts) == PBF_LAUNCHES[staged], counts   # one of the two may measure


@pytest.mark.parametrize("method", ["wcsph", "pcisph", "dfsph"])
@pytest.mark.parametrize("ratio,staged", [(2.0, True), (2.4, False)])
def test_sph_follows_too(method, ratio, staged):
    scene = lattice(27000, ratio, dt=scenes.SPH_DT)
    scene.sph = scenes.sph_parameter_arrays(scene, method=method)
    out, launches = {}, {}
    for scan in (0, 4):
        solver, state, control, params = sph.solver_for_scene(scene, sph.Method[method])
        solver.launch_shape = pbf.LaunchShape(scan, 128, 128)
        out[scan], launches[scan] = steps(solver, state, control, params, 3)
    assert launches[4][1:] == [n - (1 if staged else 0) for n in launches[0][1:]]
    for a, b in zip(out[0], out[4]):
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32))


@pytest.mark.parametrize("ratio,staged", [(2.0, True), (2.3, False)])
def test_differentiable_steps_follow_too(ratio, staged):
    scene = lattice(81 ** 3, ratio)
    outs = []
    for shape in (0, 4):
        solver, state, control, params = pbf.solver_for_scene(scene, mode=pbf.ExecutionMode.differentiable)
        solver.launch_shape = pbf.LaunchShape(shape, 128, 128)
        out, launches = steps(solver, state, control, params, 2)
        if shape == 4:
            assert launches[1] == PBF_LAUNCHES[staged]
        outs.append(out)
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32))


@pytest.mark.parametrize("count,staged", [(8000, True), (185193, False)])
def test_radii_outside_the_packed_range_stay_per_lane(count, staged):
    """Except with four lanes a particle, where the staged passes are faster all the same."""
    scene = lattice(count, 2.0, h=0.0005, dt=1e-5)   # a step moves the particles by 0.002 h
    out, launches = run(scene, pbf.LaunchShape(4, 128, 128), count=2)
    assert launches[1] == PBF_LAUNCHES[staged]
    for a, b in zip(out, run(scene, pbf.LaunchShape(0, 128, 128), count=2)[0]):
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32))


def sph_launches(scene, method, scan):
    scene.sph = scenes.sph_parameter_arrays(scene, method=method)
    solver, state, control, params = sph.solver_for_scene(scene, sph.Method[method])
    solver.launch_shape = pbf.LaunchShape(scan, 128, 128)
    return steps(solver, state, control, params, 2)[1][1]


@pytest.mark.parametrize("method", ["wcsph", "dfsph"])
def test_sph_radii_outside_the_packed_range_stay_per_lane(method):
    scene = lattice(8000, 2.0, h=0.0005, dt=4e-6)
    assert sph_launches(scene, method, 4) == sph_launches(scene, method, 0)


@pytest.mark.parametrize("count,staged", [(91125, True), (125000, False), (216000, False), (287496, True)])
def test_wcsph_between_the_waves_stays_per_lane(count, staged):
    """The staged scan's second wave begins at 113,664 particles, the per-lane scan's at 227,328."""
    scene = lattice(count, 2.0, dt=scenes.SPH_DT)
    assert sph_launches(scene, "wcsph", 4) == sph_launches(scene, "wcsph", 0) - (1 if staged else 0)


def test_autotune_leaves_the_staged_passes_their_block_size():
    """At 8,000 particles they are twice as fast as any other shape, and ignore the gather block size."""
    solver, state, control, params = pbf.solver_for_scene(lattice(8000, 2.0))
    shape, ms = solver.autotune(state, control, params, repeats=2)
    assert shape == pbf.LaunchShape(4, 128, 128) and ms > 0.0


def test_a_solver_starts_unmeasured():
    """Also where it takes the place of a solver whose particles did not fit, and among more solvers than can measure."""
    _, launches = run(lattice(8000, 2.4), pbf.LaunchShape(4, 128, 128))
    assert launches[1] == PBF_LAUNCHES[False]
    made = pbf.solver_for_scene(lattice(8000, 2.0))
    scene, others = lattice(27, 2.0), []
    assert steps(*made, 2)[1][1] == PBF_LAUNCHES[True]
    for _ in range(520):
        others.append(pbf.solver_for_scene(scene))
    for solver in (others[0], others[-1]):
        assert steps(*solver, 3)[1][1:] == [PBF_LAUNCHES[True]] * 2
    assert steps(*made, 2)[1][1] == PBF_LAUNCHES[True]
