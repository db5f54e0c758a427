"""Scenes whose support holds more particles than a list (h = 2.9 to 3.5 spacings): the
step with the lists and kernels chosen for them against the oracle, with the bounds of
test_gpu_single_scale and of test_xsph, at sizes on both sides of the density pass's
forms; equal to the batched step bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O
from sph2s_final_gb300 import scenes
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import Solver
from test_gpu_single_scale import check_step_against_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [2.8, 2.9, 3.0, 3.5])
@pytest.mark.parametrize("side", [12, 27])  # nine lanes to a particle in the density pass, and one
def test_step(side, h):
    sc = scenes.dam_break(0.5 / side, (side, side, side), dt=1e-5, h_over_s=h)
    rng = np.random.default_rng(side)
    v = rng.normal(0, 0.1, sc.fluid.positions.shape).astype(np.float32)
    b = sc.boundary.positions
    with Solver(sc.fluid, sc.boundary, sc.config, velocities=v) as s, \
            Batch([(sc.fluid.positions, b, sc.config, v)] * 2) as bt:
        for steps in (0, 3):
            s.advance(sc.dt, steps)
            check_step_against_oracle(s, sc.config, b)
        bt.advance(sc.dt, 3)
        got = bt.scene(1)
        np.testing.assert_array_equal(got["x"], s.positions())
        np.testing.assert_array_equal(got["v"], s.velocities())
        np.testing.assert_array_equal(got["rho"], s.densities())
        # the step's own force kernel, from the state that the debug pass was compared at
        x0, v0 = s.positions("by_id"), s.velocities("by_id")
        s.advance(sc.dt, 1)
        ro = O.SSRollout(sc.config, x0, b, v0)
        ro.advance(sc.dt, 1)
        st = ro.state()
        dv = np.abs(s.velocities("by_id")[st["ids"]] - st["v"]).max()
        assert dv <= 1e-5 * max(1.0, np.abs(st["v"]).max())


@pytest.mark.parametrize("dims", [(64, 64, 63), (64, 64, 64), (64, 64, 65)])
def test_equal_to_the_batched_step(dims):
    sc = scenes.dam_break(1 / 128, dims, dt=1e-5, h_over_s=3.0, border=2)
    with Solver(sc.fluid, sc.boundary, sc.config) as s, \
            Batch([(sc.fluid.positions, sc.boundary.positions, sc.config)]) as b:
        s.advance(sc.dt, 3)
        b.advance(sc.dt, 3)
        np.testing.assert_array_equal(b.scene(0)["x"], s.positions())
        np.testing.assert_array_equal(b.scene(0)["v"], s.velocities())
