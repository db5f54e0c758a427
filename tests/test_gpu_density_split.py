"""The density pass with several lanes to a particle (below 16,384 particles):
counts around a warp's three and a block's twelve particles and on both sides of
the limit, and clusters that overflow a lane's share or the list, against the
batched solver, which takes one lane to a particle.  Equal bit for bit."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import ParticleData, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cluster", [(1, 0), (2, 0), (3, 0), (4, 0), (11, 0), (12, 0), (13, 0),
                                       (2000, 39), (2000, 41), (2000, 95), (2000, 300),
                                       (16383, 50), (16384, 50)])
def test_split_density_equals_one_lane(n, cluster):
    sc = scenes.dam_break(1 / 64, (32, 32, 24))
    x = sc.fluid.positions[:n].copy()
    rng = np.random.default_rng(cluster)
    if cluster:  # within half a support radius of one particle
        x[5:5 + cluster] = x[n // 2] + rng.uniform(-0.2, 0.2, (cluster, 3)) / 64
    x = x.astype(np.float32)
    with Solver(ParticleData(x), sc.boundary, sc.config) as s, \
            Batch([(x, sc.boundary.positions, sc.config)]) as b:
        for steps in (1, 2):
            s.advance(1e-6, steps)
            b.advance(1e-6, steps)
            r = b.scene(0)
            np.testing.assert_array_equal(s.densities(), r["rho"])
            np.testing.assert_array_equal(s.positions(), r["x"])
            np.testing.assert_array_equal(s.velocities(), r["v"])
