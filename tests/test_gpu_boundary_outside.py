"""Particles at and just beyond the walls: the boundary pass walks the home
cell's candidate list up to 0.008 h outside the grid's box and scans the stencil
from there on.  On both sides of that limit, through faces, edges and corners of
both ends of the box, its step equals the debug fields' accelerations, whose
boundary sums always scan the stencil: bit for bit."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300.solver import ParticleData, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out", [0.0, 1e-4, 0.002, 0.004, 0.00799, 0.00801, 0.0101, 0.05, 0.7])
@pytest.mark.parametrize("far", [False, True])
def test_step_beyond_the_wall_equals_the_scan(out, far):
    sc = scenes.dam_break(1 / 32, (8, 8, 8))
    h, dt = 2.0 / 32, np.float32(1e-4)
    rng = np.random.default_rng(3)
    x = rng.uniform(0.05, 0.95, (900, 3))
    for k in range(900):  # a face, an edge or a corner
        axes = rng.choice(3, size=1 + k % 3, replace=False)
        x[k, axes] = (1.0 + out * h / len(axes)) if far else -out * h / len(axes)
    x = x.astype(np.float32)
    with Solver(ParticleData(x), sc.boundary, sc.config) as s:
        f = s.debug_step_fields()
        s.advance(float(dt), 1)
        assert f["nbr_boundary"].sum() > 900
        v = np.empty((900, 3), np.float32)
        v[f["ids"]] = dt * f["acc"]
        np.testing.assert_array_equal(s.velocities("by_id"), v)
