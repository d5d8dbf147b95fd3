"""The cell-offset scan on both sides of the tile count at which a block stops adding up the tiles before its own
(1024 tiles of 4096 cells, physica_b200/csrc/grid.cu): particles far from the far walls take the same steps, bit
for bit, in a domain of any size, and the step counter moves the box the same way."""
import dataclasses

import numpy as np
import pytest
import torch

from physica_b200 import pbf, scenes

pytestmark = pytest.mark.gpu


def run(cells):
    s = scenes.dam_break((9, 10, 11), (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), 5, 3, velocity_sigma=0.3)
    s = dataclasses.replace(s, box_max=tuple(float(np.float32(c * s.support_radius)) for c in cells), box_velocity=(0.05, -0.02, 0.03))
    solver, state, control, params = pbf.solver_for_scene(s)
    cache, following = solver.allocate_step_cache(), solver.allocate_state()
    for _ in range(4):
        solver.forward_step(state, control, params, following, cache)
        state, following = following, state
    out = [state.positions, state.velocities, cache.read(pbf.CacheField.NEIGHBOR_COUNTS)]
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in out]


@pytest.mark.parametrize("cells", [(40, 44, 36), (69, 89, 683), (69, 89, 684), (170, 171, 172)])
def test_steps_do_not_depend_on_the_grid(cells):
    for a, b in zip(run((24, 24, 24)), run(cells)):
        np.testing.assert_array_equal(a, b)
