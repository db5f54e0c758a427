"""Particles around the capacity of a neighbour list (96 entries; more rescan the
stencil): neighbour counts bit-exact and accelerations <= 1e-5 max-norm relative
against the oracle, and a batched scene equal to the solver bit for bit, with the
crowd alone and in an ordinary scene."""
import numpy as np
import pytest

from oracle import oracle as O
from sph2s_final_gb300 import scenes
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import ParticleData, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crowd", [64, 65, 66, 95, 96, 97, 98, 130])
@pytest.mark.parametrize("alone", [True, False])
def test_crowd(crowd, alone):
    sc = scenes.small_scene(8)
    rng = np.random.default_rng(crowd)
    h = float(sc.config.effective_radius)
    # every pair of the ball within h: each of its particles has crowd - 1 neighbours
    ball = (np.float32([0.72, 0.7, 0.71]) +
            rng.uniform(-0.25, 0.25, (crowd, 3)) * h).astype(np.float32)
    x = ball if alone else np.concatenate([sc.fluid.positions, ball])
    v = rng.normal(0, 0.2, x.shape).astype(np.float32)
    b = sc.boundary.positions
    with Solver(ParticleData(x), ParticleData(b), sc.config, velocities=v) as s, \
            Batch([(x, b, sc.config, v), (x[:5], b, sc.config)]) as bt:
        d = s.debug_step_fields()
        f = O.ss_fields(sc.config, x, v, b)
        ids = d["ids"]
        np.testing.assert_array_equal(d["nbr_fluid"], f["nbr_fluid"][ids])
        assert d["nbr_fluid"].max() == crowd  # itself included
        acc = f["acc"][ids]
        assert np.abs(d["acc"] - acc).max() <= 1e-5 * np.abs(acc).max()
        s.advance(1e-6, 2)
        bt.advance(1e-6, 2)
        got = bt.scene(0, "by_id")
        np.testing.assert_array_equal(got["x"], s.positions("by_id"))
        np.testing.assert_array_equal(got["v"], s.velocities("by_id"))
