"""A batch from 524,288 particles on sorts coherently; the solvers of its scenes,
each smaller, sort from scratch.  Steps, and a rollout whose last segment is recorded
(neighbour tables redirected into the tape), agree with them bit for bit."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300.autograd import node_grid
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import Solver

pytestmark = pytest.mark.gpu

COHERENT = 1 << 19  # kCoherentMinParticles


@pytest.fixture(scope="module")
def scs():
    out = scenes.batched_scenes(num=8, seed=11, n_min=70000, n_max=90000)
    sizes = [s.fluid.num_particles for s in out]
    assert sum(sizes) >= COHERENT > max(sizes)
    return out


def items(scs):
    return [(s.fluid.positions, s.boundary.positions, s.config) for s in scs]


def test_steps(scs):
    dt, steps = scs[0].dt, 40
    with Batch(items(scs)) as b:
        b.advance(dt, steps)
        for k, sc in enumerate(scs):
            got = b.scene(k)
            with Solver(sc.fluid, sc.boundary, sc.config) as s:
                s.advance(dt, steps)
                np.testing.assert_array_equal(got["x"], s.positions())
                np.testing.assert_array_equal(got["v"], s.velocities())
                np.testing.assert_array_equal(got["rho"], s.densities())


@pytest.mark.parametrize("every", [2, 3, 5])
def test_rollout(scs, every):
    dt, steps, rng = scs[0].dt, 5, np.random.default_rng(every)
    v0 = [rng.normal(0, 0.3, s.fluid.positions.shape).astype(np.float32) for s in scs]
    nodes = node_grid((16, 16, 16))
    target = rng.uniform(0, 800, 16 ** 3).astype(np.float32)
    with Batch(items(scs)) as b:
        b.rollout_forward(v0, None, dt, steps, every)
        end = [b.scene(k) for k in range(len(scs))]
        b.rollout_density_loss([nodes] * len(scs), [target] * len(scs))
        first = b.rollout_backward()
        second = b.rollout_backward()  # the recorded segment was overwritten: computed again
        b.advance(dt, 2)  # and steps go on from where the backward pass left the batch
        after = [b.scene(k)["x"] for k in range(len(scs))]
    for k, sc in enumerate(scs):
        with Solver(sc.fluid, sc.boundary, sc.config) as s:
            s.rollout_forward(v0[k], sc.config.viscosity, dt, steps, every)
            np.testing.assert_array_equal(end[k]["x"], s.positions())
            np.testing.assert_array_equal(end[k]["rho"], s.densities())
            s.rollout_density_loss(nodes, target)
            gv, gx, gmu = s.rollout_backward()
            s.advance(dt, 2)
            np.testing.assert_array_equal(after[k], s.positions())
        for g in (first, second):
            np.testing.assert_array_equal(g[0][k], gv)
            np.testing.assert_array_equal(g[1][k], gx)
            assert g[2][k] == gmu
