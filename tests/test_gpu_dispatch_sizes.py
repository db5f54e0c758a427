"""Solvers on both sides of the sizes at which the force pass gathers one neighbour
at a time (2^17) and the density pass is no longer launched dependent (2^20).  The
batched step of the same scene takes the other side's kernels at every size, so it
has to agree bit for bit on both."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import ParticleData, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dims,inv", [
    (131071, (64, 64, 32), 128), (131072, (64, 64, 32), 128), (131073, (64, 64, 33), 128),
    (1048575, (128, 128, 64), 192), (1048576, (128, 128, 64), 192), (1048577, (128, 128, 65), 192)])
def test_equal_to_the_batched_step(n, dims, inv):
    sc = scenes.dam_break(1 / inv, dims, dt=2.5e-5, border=1)
    x = sc.fluid.positions[:n]
    assert len(x) == n
    v = np.random.default_rng(n).normal(0, 0.2, x.shape).astype(np.float32)
    with Solver(ParticleData(x), sc.boundary, sc.config, velocities=v) as s, \
            Batch([(x, sc.boundary.positions, sc.config, v)]) as b:
        s.advance(sc.dt, 6)
        b.advance(sc.dt, 6)
        got = b.scene(0)
        np.testing.assert_array_equal(got["x"], s.positions())
        np.testing.assert_array_equal(got["v"], s.velocities())
        np.testing.assert_array_equal(got["rho"], s.densities())
