"""The staged forward passes (launch-shape variant 4, physica_b200/csrc/staged.cu) against the per-lane
passes (variant 0), bit for bit: the same sums in the same order, so any difference is a fault."""
import dataclasses

import numpy as np
import pytest
import torch

from physica_b200 import pbf, scenes

pytestmark = pytest.mark.gpu

PER_LANE, STAGED = pbf.LaunchShape(0, 128, 128), pbf.LaunchShape(4, 128, 128)


def run(scene, shape, steps, fields=True):
    solver, state, control, params = pbf.solver_for_scene(scene)
    solver.launch_shape = shape
    cache, following = solver.allocate_step_cache(), solver.allocate_state()
    out = []
    for _ in range(steps):
        solver.forward_step(state, control, params, following, cache)
        out += [following.positions.clone(), following.velocities.clone()]
        for field in (pbf.CacheField.FIRST_DENSITIES, pbf.CacheField.FIRST_LAMBDAS, pbf.CacheField.NEIGHBOR_COUNTS,
                      pbf.CacheField.VORTICITY_MAGNITUDES, pbf.CacheField.VORTICITY_NORMALS, pbf.CacheField.CONFINED_VELOCITIES,
                      pbf.CacheField.CORRECTED_POSITIONS, pbf.CacheField.RECONSTRUCTED_VELOCITIES) if fields else ():
            out.append(cache.read(field))
        state, following = following, state
    solver.synchronize()
    return [t.cpu().numpy() for t in out]


def check(scene, steps=3, **options):
    for a, b in zip(run(scene, PER_LANE, steps, **options), run(scene, STAGED, steps, **options)):
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32))


def block(count, seed=1, iterations=3, **options):
    """`count` particles of a lattice block in motion."""
    n = int(np.ceil(count ** (1 / 3)))
    s = scenes.dam_break((n, n, n), (0.0, 0.0, 0.0), (2.5 * n * 0.0125 + 0.05,) * 3, seed, iterations, velocity_sigma=0.5, **options)
    keep = {f.name: getattr(s, f.name)[..., :count] for f in dataclasses.fields(s)
            if isinstance(getattr(s, f.name), np.ndarray)}
    return dataclasses.replace(s, **{k: np.ascontiguousarray(v) for k, v in keep.items()})


# staged with four lanes per particle up to 20480 particles, blocks of 32; with one lane above 170496,
# blocks of 128; the per-lane passes between
@pytest.mark.parametrize("count", [1, 2, 31, 33, 127, 128, 129, 255, 257, 1000, 4097, 20480, 20481, 170496, 170497, 170625])
def test_counts_around_the_block(count):
    check(block(count))


@pytest.mark.parametrize("count,staged", [(20480, True), (20481, False), (170496, False), (170497, True)])
def test_sizes_choose_the_passes(count, staged):
    """The staged step has one kernel less: its post-loop scan is part of the vorticity pass."""
    scene = block(count, iterations=3)
    solver, state, control, params = pbf.solver_for_scene(scene)
    cache, following = solver.allocate_step_cache(), solver.allocate_state()
    for k in range(2):
        before = pbf.launch_count()
        solver.forward_step(state, control, params, following, cache)
        launches = pbf.launch_count() - before
        state, following = following, state
    assert launches == (15 if staged else 16)


@pytest.mark.parametrize("iterations", [0, 3])
@pytest.mark.parametrize("kind", ["block", "spray", "crowded", "coincident"])
def test_hit_mask_lists(kind, iterations):
    """From 140,001 to 170,496 particles variant 4 runs the per-lane passes over hit masks."""
    n = 140001 + iterations
    s = block(n, seed=14, iterations=iterations)
    rng = np.random.default_rng(15)
    if kind == "spray":
        fly = rng.permutation(n)[:n // 9]
        s.positions[:, fly] = (rng.random((3, n // 9)) * np.asarray(s.box_max)[:, None]).astype(np.float32)
    if kind == "crowded":   # up to 3,000 candidates: more than 48 masks
        s.positions[:, :3000] = (0.2 + 0.06 * rng.random((3, 3000))).astype(np.float32)
    if kind == "coincident":
        s.positions[:, 100:200], s.velocities[:, 100:200] = s.positions[:, 200:300], s.velocities[:, 200:300]
        s.masses[:] *= rng.choice([0.5, 1.0], n).astype(np.float32)
    check(s, steps=2, fields=iterations > 0)


@pytest.mark.parametrize("count,steps", [(13824, 100), (175616, 25)])
def test_long_runs(count, steps):
    """A falling, splashing block, with four lanes a particle and with one."""
    scene = block(count, seed=13, iterations=4)
    out = []
    for shape in (PER_LANE, STAGED):
        solver, state, control, params = pbf.solver_for_scene(scene)
        solver.launch_shape = shape
        cache, following = solver.allocate_step_cache(), solver.allocate_state()
        before = pbf.launch_count()
        for _ in range(steps):
            solver.forward_step(state, control, params, following, cache)
            state, following = following, state
        out.append([state.positions.cpu().numpy(), state.velocities.cpu().numpy()])
        launches = pbf.launch_count() - before
    assert launches < 17.5 * steps   # 17 a staged step and 18 a per-lane one: most were staged
    for a, b in zip(*out):
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32))


@pytest.mark.parametrize("count", [8000, 180000])
def test_spray_whose_windows_exceed_the_stage(count):
    """Thin spray beside and above a dense block: its blocks' windows cover the block's columns."""
    s = block(count)
    rng = np.random.default_rng(3)
    fly = rng.permutation(count)[:count // 9]
    s.positions[:, fly] = (rng.random((3, count // 9)) * np.asarray(s.box_max)[:, None]).astype(np.float32)
    check(s)


@pytest.mark.parametrize("count", [3000, 180000])
def test_crowded_lists_overflow(count):
    s = block(count)
    s.positions[:, :3000] = (0.2 + 0.06 * np.random.default_rng(4).random((3, 3000))).astype(np.float32)
    check(s, steps=2)


@pytest.mark.parametrize("count", [2000, 180000])
@pytest.mark.parametrize("strength", [0.0, 1e-5])
def test_mixed_masses_and_coincident_particles(strength, count):
    s = block(count, seed=5)
    rng = np.random.default_rng(6)
    s.masses[:] *= rng.choice([0.5, 1.0, 1.5], count).astype(np.float32)
    s.rest_densities[:] *= rng.choice([0.8, 1.0], count).astype(np.float32)
    s.artificial_pressure_strength[:] = strength
    s.positions[:, 100:110] = s.positions[:, 110:120]
    s.velocities[:, 100:110] = s.velocities[:, 110:120]
    s.positions[:, 200:210] = s.positions[:, 210:220] + np.float32(1e-12)
    check(s)


@pytest.mark.parametrize("n", [9, 56])
@pytest.mark.parametrize("h", [0.0008, 0.003, 1.0, 3000.0])
def test_support_radii_inside_and_outside_the_packed_range(h, n):
    """The packed pair arithmetic covers radii from 2^-10 to 2^10; others take the scalar path."""
    spacing = 0.5 * h
    s = scenes.dam_break((n, n, n), (0.0, 0.0, 0.0), ((n + 3) * spacing,) * 3, 7, 3, h=h, velocity_sigma=0.2 * h)
    check(s, steps=2)


@pytest.mark.parametrize("count", [4000, 180000])
def test_moving_box(count):
    """Six steps of a moving box (particles whose sort and gather cells differ: below)."""
    s = dataclasses.replace(block(count, seed=8), box_velocity=(0.37, -0.11, 0.23))
    check(s, steps=6)


def fma32(a, b, c):
    """float32 fma(a, b, c): the product is exact in float64."""
    return np.float32(np.float64(a) * np.float64(b) + np.float64(c))


def straddled(s, step, per_axis, seed):
    """Moves `per_axis` particles of the resting scene `s` an axis in x and y onto the floats beside their nearest cell
    boundary at the time of `step`, and counts, as grid.cu evaluates them, those whose sort cell and gather cell
    there differ."""
    rng = np.random.default_rng(seed)
    h, time = np.float32(s.support_radius), np.float32(np.float32(step) * np.float32(s.time_step))
    differ = 0
    for axis in (0, 1):
        low, speed = np.float32(s.box_min[axis]), np.float32(s.box_velocity[axis])
        origin = fma32(time, speed, low)
        x = s.positions[axis]
        move = rng.permutation(s.count)[:per_axis]
        k = np.rint((x[move].astype(np.float64) - origin) / h)
        y = (np.float64(origin) + k * np.float64(h)).astype(np.float32)
        side = rng.integers(-1, 2, per_axis)
        y = np.where(side < 0, np.nextafter(y, np.float32(-1e9)), np.where(side > 0, np.nextafter(y, np.float32(1e9)), y))
        x[move] = y
        sort_cell = np.floor(fma32(-time, speed, (y - low).astype(np.float32)).astype(np.float32) / h)
        gather_cell = np.floor((y - origin).astype(np.float32) / h)
        differ += int((sort_cell != gather_cell).sum())
    return differ


@pytest.mark.parametrize("lattice,box_z", [((36, 36, 4), 0.06), ((210, 210, 4), 0.06), ((36, 36, 14), 0.2)])
def test_sort_cell_and_gather_cell_differ(lattice, box_z):
    """In a moving box the two cell formulas round differently; a particle on a cell boundary is then sorted into another
    stencil column than its own.  The grid has few cells in z, so that a block's windows still cover that column:
    the particle must find itself there (neighbour counts leave it out)."""
    low = (37.0, -21.0, 0.0)
    s = scenes.dam_break(lattice, low, (low[0] + 6.0, low[1] + 6.0, box_z), 8, 2, gravity=(0.0, 0.0, 0.0))
    s = dataclasses.replace(s, box_velocity=(0.37, -0.11, 0.0))
    assert straddled(s, 1, s.count // 8, 9) > s.count // 100
    check(s, steps=1)


@pytest.mark.parametrize("count", [40, 4000, 180000])
def test_values_that_are_not_finite(count):
    """Pairs without a kernel term (coincident particles here) add nothing, whatever else they hold: an infinite mass,
    the infinite velocity of a particle that came from infinity."""
    s = block(count, seed=12)
    for i in (10, 20):
        s.positions[:, i + 1], s.velocities[:, i + 1] = s.positions[:, i], s.velocities[:, i]
    s.masses[10] = np.inf
    s.positions[1, 30:32], s.velocities[:, 30:32] = np.inf, 0.0      # clamped to the top of the box
    s.positions[::2, 31] = s.positions[::2, 30]
    for a, b in zip(run(s, PER_LANE, 1), run(s, STAGED, 1)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("kind", ["block", "spray", "crowded"])
def test_differentiable_steps_record_the_same_lists(kind, recompute):
    """Adjoint and tangent over the lists of sorted slots that the staged passes store (differentiable
    steps use the staged passes from 2^19 particles on)."""
    n = (1 << 19) + 77
    s = block(n, seed=9, iterations=2)
    rng = np.random.default_rng(10)
    if kind == "spray":
        fly = rng.permutation(n)[:20000]
        s.positions[:, fly] = (rng.random((3, 20000)) * np.asarray(s.box_max)[:, None]).astype(np.float32)
    if kind == "crowded":
        s.positions[:, :3000] = (0.2 + 0.06 * rng.random((3, 3000))).astype(np.float32)
    out = []
    for shape in (PER_LANE, STAGED):
        solver, state, control, params = pbf.solver_for_scene(s, mode=pbf.ExecutionMode.differentiable)
        solver.launch_shape = shape
        solver.set_checkpoint_recompute(recompute)
        cache, following = solver.allocate_step_cache(), solver.allocate_state()
        solver.forward_step(state, control, params, following, cache)
        g = torch.Generator(device="cuda").manual_seed(11)
        rand = lambda dtype: torch.randn((3, s.count), generator=g, device="cuda", dtype=dtype)
        pa, ca, qa = solver.allocate_state_adjoint(), solver.allocate_control_adjoint(), solver.allocate_parameter_adjoint()
        solver.vjp_step(state, control, params, following, cache, pbf.StateAdjoint(rand(torch.float64), rand(torch.float64)), pa,
                        ca, qa)
        tangent = solver.allocate_state_tangent()
        solver.jvp_step(state, control, params, following, cache, pbf.StateTangent(rand(torch.float32), rand(torch.float32)),
                        pbf.Control(rand(torch.float32)), solver.allocate_parameter_tangent(), tangent)
        solver.synchronize()
        out.append([following.positions, following.velocities, pa.positions, pa.velocities, ca.external_accelerations,
                    tangent.positions, tangent.velocities, *qa.tensors.values()])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())


@pytest.mark.parametrize("counts", [(65, 700, 3, 1, 2049, 130), (65, 90001, 3, 1, 2049, 80000)])
def test_batch_blocks_span_scenes(counts):
    parts = [scenes.batched_scene(c, 40 + k, 3, velocity_sigma=0.3) for k, c in enumerate(counts)]
    results = []
    for shape in (PER_LANE, STAGED):
        batch, state, control, params = pbf.batch_for_scenes(parts)
        batch.launch_shape = shape
        batch.reserve_caches(1)
        following = batch.allocate_state()
        for _ in range(3):
            batch.forward_step(state, control, params, following, 0)
            state, following = following, state
        torch.cuda.synchronize()
        results.append((state.positions.cpu().numpy(), state.velocities.cpu().numpy()))
    for a, b in zip(*results):
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32))
