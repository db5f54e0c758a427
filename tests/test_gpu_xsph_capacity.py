"""XSPH with particles around the capacity of a neighbour list (96 entries), in one
crowd and with coincident pairs inside it: one step against the oracle with the
bounds of test_xsph, where the particles of the crowd rescan the stencil in the force
pass and in the XSPH pass."""
import numpy as np
import pytest

from oracle import oracle as O
from sph2s_final_gb300 import scenes
from sph2s_final_gb300.solver import ParticleData, Solver
from test_xsph import gpu_vs_oracle

pytestmark = pytest.mark.gpu

CAPACITY = 96


@pytest.mark.parametrize("crowd", [96, 97, 98, 99, 130])
@pytest.mark.parametrize("coincident", [False, True])
def test_crowd(crowd, coincident):
    sc = scenes.small_scene(8)
    rng = np.random.default_rng(crowd)
    h = float(sc.config.effective_radius)
    # every pair of the ball within h: each of its particles has crowd - 1 neighbours
    ball = (np.float32([0.72, 0.7, 0.71]) +
            rng.uniform(-0.25, 0.25, (crowd, 3)) * h).astype(np.float32)
    if coincident:
        ball[5] = ball[6]
        ball[40] = ball[41]
    x = np.concatenate([sc.fluid.positions, ball])
    v = rng.normal(0, 0.3, x.shape).astype(np.float32)
    b = sc.boundary.positions
    with Solver(ParticleData(x), ParticleData(b), sc.config) as s:
        # counted with the particle itself and those at distance 0, which are not listed
        nbr = s.debug_step_fields()["nbr_fluid"].max() - 1
    assert nbr == crowd - 1 and (nbr > CAPACITY) == (crowd > 97)
    dx, dv = gpu_vs_oracle(sc.config, x, v, b, 1e-5, 0.7)
    assert dx <= 1e-6 and dv <= 1e-5, (dx, dv)
