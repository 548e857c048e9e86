"""GPU checks of the water step's gather where many particles share a node's bins: as many as a thread keeps, as it
orders alone and one more of each, crowds among many other particles, a box full of particles, and the time a crowd takes.
Bit-exact against the snapshot oracle."""
import dataclasses

import numpy as np
import pytest

from neonengine_b200.water_synth import WaterConfig
from test_water_lists_gpu import _check

pytestmark = pytest.mark.gpu


def _positions(cfg, crowd, sigma, seed):
    """A crowd of particles around the box's centre, the others anywhere, their ids in random order."""
    rng = np.random.default_rng(seed)
    lo, hi = np.array(cfg.box_min), np.array(cfg.box_max)
    pos = np.ones((cfg.n_particles, 4), np.float32)
    pos[:, :3] = lo + (0.1 + 0.8 * rng.random((cfg.n_particles, 3))) * (hi - lo)
    pos[:crowd, :3] = (lo + hi) / 2 + sigma * rng.standard_normal((crowd, 3))
    return np.ascontiguousarray(pos[rng.permutation(cfg.n_particles)])


@pytest.mark.parametrize("crowd", [32, 33, 64, 97, 128, 129, 130, 700])
@pytest.mark.parametrize("sigma", [0.0, 0.01, 0.08])
def test_crowds(crowd, sigma):
    cfg = WaterConfig(particles_per_side=9, box_min=(0.0, 0.0, 0.0), box_max=(1.6, 1.2, 1.4), collision_substeps=0, jacobi_iterations=4)
    _check(cfg, _positions(cfg, crowd, sigma, crowd), 1)
    _check(dataclasses.replace(cfg, collision_substeps=2), _positions(cfg, crowd, sigma, crowd + 1), 2)


@pytest.mark.parametrize("crowd,sigma", [(40, 0.0), (57, 0.0), (62, 0.0), (400, 0.03), (20000, 0.2)])
def test_crowds_among_many(crowd, sigma):
    cfg = WaterConfig(particles_per_side=42, collision_substeps=0, jacobi_iterations=2)
    _check(cfg, _positions(cfg, crowd, sigma, 5), 1)


@pytest.mark.parametrize("side", [10, 13])
def test_full_box(side):
    """About as many particles a cell as the separation's list and a thread's share of the gather hold, and twice that."""
    cfg = WaterConfig(particles_per_side=side, box_min=(0.0, 0.0, 0.0), box_max=(0.7, 0.8, 0.6), collision_substeps=2, jacobi_iterations=3)
    _check(cfg, _positions(cfg, 0, 0.0, 2), 3)


def test_a_crowd_takes_no_walk_for_every_particle():
    import torch
    from neonengine_b200.water_physics import WaterPhysics
    cfg = WaterConfig(particles_per_side=10, collision_substeps=1)
    pos = _positions(cfg, 1000, 0.0, 1)
    sim = WaterPhysics(cfg, pos)
    ms = []
    for _ in range(4):  # the first step builds its graph
        sim.set_particles(pos)
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        start.record()
        sim.run_simulation(1, stream=torch.cuda.current_stream())
        end.record()
        torch.cuda.synchronize()
        ms.append(start.elapsed_time(end))
    sim.close()
    assert min(ms) < 20.0, ms  # a walk of the lists for every particle took 135 ms, sorting the particles in memory 23


def test_a_crowd_beyond_the_list_ends_the_walk():
    from neonengine_b200.water_physics import WaterPhysics
    cfg = WaterConfig(particles_per_side=10, collision_substeps=1)
    pos = _positions(cfg, 1000, 0.0, 1)
    sim = WaterPhysics(cfg, pos)
    ms = []
    for _ in range(6):
        sim.set_particles(pos)
        ms.append(sim.profile_step()["separate"])
    sim.close()
    assert min(ms) < 0.12, ms  # walking lists of 1000 to their end took 0.22 ms, stopping when 128 are found 0.05
