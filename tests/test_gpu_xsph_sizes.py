"""XSPH step against the oracle at sizes around the 256-thread blocks and for
blocks that touch one, two or three walls (the boundary force comes from its own
pass): positions <= 1e-6 and velocities <= 1e-5 relative, the bounds of the
XSPH step at its ordinary size."""
import numpy as np
import pytest

from oracle import oracle as O
from sph2s_final_gb300 import scenes
from sph2s_final_gb300.solver import ParticleData, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 3, 17), (16, 16, 1), (257, 1, 1), (13, 14, 15),
                                  (16, 32, 9)])
@pytest.mark.parametrize("shift", [0.0, 0.3])
def test_xsph_step_sizes(dims, shift):
    sc = scenes.dam_break(1 / 32 if max(dims) <= 32 else 1 / 320, dims, seed=4, dt=2e-5)
    x = sc.fluid.positions + np.float32([0.0, shift, 0.0])
    v = np.random.default_rng(5).normal(0, 0.2, x.shape).astype(np.float32)
    sc.config.xsph_coeff = 0.4
    with Solver(ParticleData(x), sc.boundary, sc.config, velocities=v) as s:
        s.set_integrator("xsph")
        s.advance(sc.dt, 1)
        xg, vg = s.positions("by_id"), s.velocities("by_id")
    xo, vo = O.ss_xsph_step(sc.config, x, v, sc.boundary.positions, sc.dt, 0.4)
    assert np.abs(xg - xo).max() <= 1e-6
    assert np.abs(vg - vo).max() <= 1e-5 * max(1.0, np.abs(vo).max())
