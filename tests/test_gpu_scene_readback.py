"""Readback of a batched scene around its 4 MiB chunks (7 floats per particle:
149,796.6 particles to a chunk; positions alone: 349,525.3): equal to the lone
solver's arrays bit for bit in both orders, whichever arrays are wanted, also
after a smaller scene was read."""
import ctypes as C

import numpy as np
import pytest

from sph2s_final_gb300._abi import check, fptr, lib
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import Grid, ParticleData, Solver, SolverConfiguration

pytestmark = pytest.mark.gpu

NONE = np.zeros((0, 3), np.float32)


@pytest.mark.parametrize("n", [1, 255, 149796, 149797, 299594, 349526])
def test_chunks(n):
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    v = rng.normal(0, 1, (n, 3)).astype(np.float32)
    g = Grid.make_grid((0, 0, 0), (1, 1, 1), 0.01)
    cfg = SolverConfiguration.direct(0.01, 1e-3, 1000.0, 30.0, 5.0, 88.1472, 0.8, g)
    with Batch([(x[:3], NONE, cfg), (x, NONE, cfg, v)]) as b, \
            Solver(ParticleData(x), None, cfg, velocities=v) as s:
        b.advance(1e-7, 1)
        s.advance(1e-7, 1)
        for order, code in (("sorted", 0), ("by_id", 1)):
            b.scene(0, order)
            got = b.scene(1, order)
            np.testing.assert_array_equal(got["x"], s.positions(order))
            np.testing.assert_array_equal(got["v"], s.velocities(order))
            np.testing.assert_array_equal(got["rho"], s.densities(order))
            only = np.empty((n, 3), np.float32)
            check(lib().sphb_get_scene(b._h, 1, fptr(only), None, None, code))
            np.testing.assert_array_equal(only, got["x"])
            rho = np.empty(n, np.float32)
            check(lib().sphb_get_scene(b._h, 1, None, None, fptr(rho), code))
            np.testing.assert_array_equal(rho, got["rho"])
            check(lib().sphb_get_scene(b._h, 1, None, None, None, code))
