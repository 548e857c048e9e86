"""GPU checks of the pressure iterations as one cooperative launch: grids beyond sixteen CTAs' shared memory, and grids
whose layers are too large for the CTAs of a cluster that the registers would allow.  Bit-exact against the snapshot
oracle and against one launch per iteration, for odd and even iteration counts."""
import numpy as np
import pytest

from neonengine_b200.water_synth import WaterConfig, spawn_particles
from oracle import water
from test_water_lists_gpu import oracle_params, pytestmark  # noqa: F401


@pytest.mark.parametrize("size", [(7.0, 6.0, 6.0), (16.0, 10.0, 0.6)])
@pytest.mark.parametrize("iterations", [6, 7])
def test_cooperative_pressure(size, iterations):
    from neonengine_b200.water_physics import WaterPhysics
    cfg = WaterConfig(particles_per_side=12, box_min=(0.0, 0.0, 0.0), box_max=size, jacobi_iterations=iterations, collision_substeps=2)
    nx, ny, nz = cfg.grid_dim
    # no cluster: too many cells for 16 CTAs, or (with two CTAs or more) fewer cells per CTA than one layer; but two cells per resident thread
    assert cfg.n_cells > 16 * 12288 or all((cfg.n_cells + s - 1) // s < nx * ny or (cfg.n_cells + s - 1) // s > 12288 for s in (16, 8, 4, 2))
    assert 12288 < cfg.n_cells <= 2 * 1024 * 148
    pos0 = spawn_particles(cfg)
    pos0[:500, :3] = np.array([size[0] / 2, size[1] / 2, size[2] / 2], np.float32) + np.random.default_rng(1).normal(0, 0.1, (500, 3)).astype(np.float32)
    steps, launches, results = 2, [], []
    for fused in (1, 0):
        sim = WaterPhysics(cfg, pos0)
        sim.set_option("fused_jacobi", fused)
        before = sim.launch_count()
        sim.run_simulation(steps)
        launches.append((sim.launch_count() - before) // steps)
        assert sim.status() == 0
        results.append((sim.read_particles(), sim.read_grids()))
        sim.close()
    assert launches[1] - launches[0] == iterations - 1
    pos, vel = pos0.copy(), np.zeros_like(pos0)
    grids = water.step(oracle_params(cfg), pos, vel, steps, collision_mode=1)
    for (gp, gv), got in results:
        np.testing.assert_array_equal(gp, pos)
        np.testing.assert_array_equal(gv, vel)
        for k, v in got.items():
            np.testing.assert_array_equal(v, grids[k], err_msg=k)
