"""The staged SPH passes (launch-shape variant 4, physica_b200/csrc/sph_staged.cu) against the per-lane
passes (variant 0), bit for bit."""
import dataclasses

import numpy as np
import pytest
import torch

from physica_b200 import pbf, scenes, sph
from test_gpu_staged import straddled

pytestmark = pytest.mark.gpu

METHODS = ["wcsph", "pcisph", "iisph", "dfsph"]


def block(count, method, seed=1, h_scale=1.0, sigma=0.3):
    n = int(np.ceil(count ** (1 / 3)))
    h = scenes.H * h_scale
    s = scenes.dam_break((n, n, n), (0.0, 0.0, 0.0), (2.5 * n * 0.5 * h + 2 * h,) * 3, seed, 0, h=h, dt=scenes.SPH_DT,
                         velocity_sigma=sigma * h_scale)
    keep = {f.name: np.ascontiguousarray(getattr(s, f.name)[..., :count]) for f in dataclasses.fields(s)
            if isinstance(getattr(s, f.name), np.ndarray)}
    s = dataclasses.replace(s, **keep)
    s.sph = scenes.sph_parameter_arrays(s, method=method)
    return s


def run(scene, method, scan, steps, mode=pbf.ExecutionMode.forward, first_step=0, warm=None):
    solver, state, control, params = sph.solver_for_scene(scene, sph.Method[method], mode=mode)
    state.step_index = first_step
    if warm is not None:
        state.warm_divergence_pressure.copy_(torch.from_numpy(warm))
        state.warm_density_pressure.copy_(torch.from_numpy(warm))
    solver.launch_shape = pbf.LaunchShape(scan, 128, 128)
    cache, following = solver.allocate_step_cache(), solver.allocate_state()
    out = []
    for _ in range(steps):
        solver.forward_step(state, control, params, following, cache)
        out += [following.positions.clone(), following.velocities.clone(), cache.read(sph.CacheField.DENSITIES)]
        if method != "wcsph":
            out.append(cache.read(sph.CacheField.PREDICTED_DENSITIES))
        if method == "dfsph":
            out += [following.warm_divergence_pressure.clone(), following.warm_density_pressure.clone()]
        if mode == pbf.ExecutionMode.differentiable:
            g = torch.Generator(device="cuda").manual_seed(3)
            na, pa = solver.allocate_state_adjoint(), solver.allocate_state_adjoint()
            na.positions.normal_(generator=g)
            na.velocities.normal_(generator=g)
            ca, qa = solver.allocate_control_adjoint(), solver.allocate_parameter_adjoint()
            solver.vjp_step(state, control, params, following, cache, na, pa, ca, qa)
            out += [pa.positions, pa.velocities, ca.external_accelerations, *qa.tensors.values()]
        state, following = following, state
    solver.synchronize()
    return [t.cpu().numpy() for t in out]


def check(scene, method, steps=3, **options):
    for a, b in zip(run(scene, method, 0, steps, **options), run(scene, method, 4, steps, **options)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("count", [1, 33, 128, 129, 3001])
def test_counts_around_the_block(method, count):
    check(block(count, method), method)


@pytest.mark.parametrize("method", METHODS)
def test_spray_coincident_particles_and_mixed_masses(method):
    s = block(4000, method, seed=2)
    rng = np.random.default_rng(3)
    fly = rng.permutation(4000)[:500]
    s.positions[:, fly] = (rng.random((3, 500)) * np.asarray(s.box_max)[:, None]).astype(np.float32)
    s.positions[:, 100:110] = s.positions[:, 110:120]
    s.sph["masses"][:] *= rng.choice([0.5, 1.0], 4000).astype(np.float32)
    check(s, method)


@pytest.mark.parametrize("method", ["pcisph", "dfsph"])
def test_displacements_beyond_the_skin(method):
    """Fast particles outrun the lists' skin: the predicted density walks the stencil."""
    check(block(2000, method, seed=4, sigma=20.0), method, steps=2)


@pytest.mark.parametrize("method", METHODS)
def test_crowded_lists_overflow(method):
    s = block(2000, method, seed=5)
    s.positions[:] = (0.2 + 0.05 * np.random.default_rng(6).random((3, 2000))).astype(np.float32)
    check(s, method, steps=1)


@pytest.mark.parametrize("h_scale", [0.03, 1.0e5])
def test_support_radii_outside_the_packed_range(h_scale):
    check(block(500, "pcisph", seed=7, h_scale=h_scale), "pcisph", steps=2)


@pytest.mark.parametrize("method", METHODS)
def test_differentiable_steps(method):
    check(block(2500, method, seed=8), method, steps=2, mode=pbf.ExecutionMode.differentiable)


@pytest.mark.parametrize("method", METHODS)
def test_sort_cell_and_gather_cell_differ(method):
    """As in test_gpu_staged.py: particles of a moving box that are sorted into another column than their own."""
    low = (37.0, -21.0, 0.0)
    s = scenes.dam_break((36, 36, 4), low, (low[0] + 6.0, low[1] + 6.0, 0.06), 8, 0, dt=scenes.SPH_DT)
    s = dataclasses.replace(s, box_velocity=(0.37, -0.11, 0.0))
    assert straddled(s, 41, s.count // 8, 9) > s.count // 100
    s.sph = scenes.sph_parameter_arrays(s, method=method)
    check(s, method, steps=1, first_step=41)


@pytest.mark.parametrize("method", METHODS)
def test_values_that_are_not_finite(method):
    """Pairs in the lists' skin, beyond the support, add nothing: neither an infinite mass nor an infinite pressure."""
    s = block(4000, method, seed=9)
    s.sph["masses"][[500, 1500]] = np.inf
    warm = np.full(4000, 10.0, np.float32)
    warm[[2500, 3500]] = np.inf, np.nan
    check(s, method, steps=1, **({"warm": warm} if method == "dfsph" else {}))


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("count", [88, 95, 96, 97, 104])
def test_lists_near_their_capacity(method, count):
    """Balls of `count` particles within each other's support, over four stencil columns so that they fit the
    hit records: a staged list holds up to 95 entries beside the particle itself, a longer one overflows."""
    s = block(4 * count, method, seed=10)
    rng = np.random.default_rng(11)
    h = s.support_radius
    for ball in range(4):
        x = rng.normal(size=(3, count))
        x *= 0.45 * h * rng.random(count) ** (1 / 3) / np.linalg.norm(x, axis=0)
        x[0], x[1] = np.abs(x[0]) * (-1.0) ** np.arange(count), np.abs(x[1]) * (-1.0) ** (np.arange(count) // 2)
        x[2] = np.abs(x[2])   # one cell in z
        s.positions[:, ball * count:(ball + 1) * count] = (x + (np.array([2, 3, 2]) + ball)[:, None] * h).astype(np.float32)
    s.box_max = (12 * h,) * 3
    check(s, method, steps=1)
