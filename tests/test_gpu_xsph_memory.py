"""XSPH switched on while the memory holds its first buffer and not its second: refused,
and switched on later with the memory there; the steps are those of a solver that had
it from the start."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300._abi import SphError
from sph2s_final_gb300.solver import Grid, ParticleData, Solver, SolverConfiguration
from test_gpu_list_memory import MiB, Short

pytestmark = pytest.mark.gpu


def test_second_buffer_refused_first():
    n = 8 << 20  # 128 MiB and 32 MiB
    x = scenes.jitter(scenes.lattice_block(1 / 256, (256, 256, 128)), 1 / 256, 0.01, 1)[:n]
    g = Grid.make_grid((0, 0, 0), (1, 1, 1), 1 / 128)
    cfg = SolverConfiguration.direct(1 / 128, 1000.0 / 256 ** 3, 1000.0, 30.0, 5.0, 88.1472, 0.8, g,
                                     epsilon=0.3)
    v = np.random.default_rng(0).normal(0, 0.1, x.shape).astype(np.float32)
    with Solver(ParticleData(x), None, cfg, velocities=v) as a, \
            Solver(ParticleData(x), None, cfg, velocities=v) as b:
        a.set_integrator("xsph")
        a.advance(1e-5, 2)
        b.sync()
        with Short(144 * MiB):
            with pytest.raises(SphError, match="SPH_E_CUDA"):
                b.set_integrator("xsph")
        b.set_integrator("xsph")
        b.advance(1e-5, 2)
        np.testing.assert_array_equal(a.positions(), b.positions())
        np.testing.assert_array_equal(a.velocities(), b.velocities())
