"""GPU parity of the water step's particle lists and pressure cluster where they can go wrong: particles crowded
beyond the separation's candidate list and the gather's id list, particles outside the box, one and five
sub-steps, grids that choose each cluster size, one-cell interiors.  Bit-exact against the snapshot oracle."""
import dataclasses
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))

pytestmark = pytest.mark.gpu

from make_water_golden import oracle_params, small_config  # noqa: E402
from neonengine_b200.water_synth import WaterConfig, spawn_particles  # noqa: E402
from oracle import water  # noqa: E402


def _check(cfg, pos0, steps):
    from neonengine_b200.water_physics import WaterPhysics
    sim = WaterPhysics(cfg, pos0)
    sim.run_simulation(steps)
    pos, vel = pos0.copy(), np.zeros_like(pos0)
    grids = water.step(oracle_params(cfg), pos, vel, steps, collision_mode=1)
    assert sim.status() == 0
    gp, gv = sim.read_particles()
    np.testing.assert_array_equal(gp, pos)
    np.testing.assert_array_equal(gv, vel)
    for k, v in sim.read_grids().items():
        np.testing.assert_array_equal(v, grids[k], err_msg=k)
    sim.close()


@pytest.mark.parametrize("substeps,iterations", [(1, 2), (5, 3), (2, 1), (3, 8)])
def test_crowded_and_outside(substeps, iterations):
    cfg = dataclasses.replace(small_config(), particles_per_side=7, collision_substeps=substeps, jacobi_iterations=iterations)
    rng = np.random.default_rng(substeps)
    pos0 = np.ones((343, 4), np.float32)
    pos0[:200, :3] = rng.normal(0.0, 0.03, (200, 3))       # 200 particles within a few cells of one another
    pos0[200:, :3] = rng.uniform(-1.4, 1.4, (143, 3))      # some of them outside the box
    pos0[7] = pos0[3]                                      # coincident: never separated
    _check(cfg, pos0, 2)


@pytest.mark.parametrize("box", [((0.0, 0.0, 0.0), (0.3, 0.3, 0.3)), ((0.0, 0.0, 0.0), (2.0, 2.0, 0.4)), ((0.0, 0.0, 0.0), (0.5, 0.4, 3.0)),
                                 ((0.0, 0.0, 0.0), (6.0, 0.3, 0.6)), ((-1.0, -1.0, -1.0), (4.3, 3.6, 3.9))])
def test_grid_shapes(box):
    cfg = WaterConfig(particles_per_side=5, box_min=box[0], box_max=box[1], jacobi_iterations=9, collision_substeps=2)
    _check(cfg, spawn_particles(cfg), 3)
