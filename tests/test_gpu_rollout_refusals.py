"""A rollout refuses a time step that is not finite, however many segments it has:
the last one is recorded rather than advanced, and is checked all the same."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300._abi import SphError
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [float("inf"), float("nan"), 0.0, -1e-4])
@pytest.mark.parametrize("every", [1, 2, 4, 9])
def test_time_step(dt, every):
    sc = scenes.small_scene(5)
    with Solver(sc.fluid, sc.boundary, sc.config) as s, \
            Batch([(sc.fluid.positions, sc.boundary.positions, sc.config)] * 2) as b:
        for call in (lambda: s.rollout_forward(None, 5.0, dt, 4, every),
                     lambda: b.rollout_forward(None, None, dt, 4, every)):
            with pytest.raises(SphError, match="SPH_E_INVALID"):
                call()
        s.rollout_forward(None, 5.0, sc.dt, 4, every)
        b.rollout_forward(None, None, sc.dt, 4, every)
        assert np.isfinite(s.positions()).all()
        np.testing.assert_array_equal(b.scene(1)["x"], s.positions())
