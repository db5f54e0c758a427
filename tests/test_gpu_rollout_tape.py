"""The rollout's forward pass records its last segment for the backward pass:
one segment, an even and a ragged last one, one step each.  The solver's state
is what its own steps leave, before and after the backward pass (which ends at
the first segment's end); gradients do not depend on the interval, on a second
backward pass or on steps taken in between.  All equal bit for bit."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300.autograd import node_grid
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import Solver

pytestmark = pytest.mark.gpu

T, MU = 7, 3.0


def same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(np.asarray(x), np.asarray(y))


def state(s):
    return s.positions(), s.velocities(), s.densities(), s.ids()


@pytest.fixture(scope="module")
def case():
    sc, v = scenes.differentiable_scene((9, 13, 11))
    sc.config.viscosity = MU
    target = np.random.default_rng(3).uniform(0, 800, 32 ** 3).astype(np.float32)
    at = {}
    with Solver(sc.fluid, sc.boundary, sc.config, v) as s:
        for k in range(1, T + 1):
            s.advance(sc.dt, 1)
            at[k] = state(s)
    with Solver(sc.fluid, sc.boundary, sc.config) as s:
        s.rollout_forward(v, MU, sc.dt, T, 1)
        s.rollout_density_loss(node_grid(), target)
        grads = s.rollout_backward()
    return sc, v, target, at, grads


@pytest.mark.parametrize("mode", ["full", "coherent"])
@pytest.mark.parametrize("every", [1, 3, 6, 7, 20])
def test_recorded_segment(case, every, mode):
    sc, v, target, at, grads = case
    with Solver(sc.fluid, sc.boundary, sc.config) as s:
        s.debug_sort_mode(mode)
        for extra in (0, 2):
            before = s.step_count
            s.rollout_forward(v, MU, sc.dt, T, every)
            assert s.step_count == before + T
            same(state(s), at[T])
            s.rollout_density_loss(node_grid(), target)
            s.advance(sc.dt, extra)
            for _ in range(2):
                same(s.rollout_backward(), grads)
                same(state(s)[:2], at[min(every, T)][:2])


@pytest.mark.parametrize("every", [3, 7])
def test_recorded_segment_of_a_batch(case, every):
    sc, v, target, at, grads = case
    with Batch([(sc.fluid.positions, sc.boundary.positions, sc.config)] * 2) as b:
        for extra in (0, 2):
            b.rollout_forward([v, v], np.full(2, MU, np.float32), sc.dt, T, every)
            for k in range(2):
                r = b.scene(k)
                same((r["x"], r["v"], r["rho"]), at[T][:3])
            b.rollout_density_loss([node_grid()] * 2, [target] * 2)
            b.advance(sc.dt, extra)
            for _ in range(2):
                g = b.rollout_backward()
                for k in range(2):
                    same((g[0][k], g[1][k], g[2][k]), grads)
                    r = b.scene(k)
                    same((r["x"], r["v"]), at[min(every, T)][:2])


def test_other_integrator_is_not_recorded(case):
    sc, v, _, _, _ = case
    ends = []
    with Solver(sc.fluid, sc.boundary, sc.config, v) as s:
        s.set_integrator("xsph")
        s.advance(sc.dt, T)
        ends.append(state(s))
    with Solver(sc.fluid, sc.boundary, sc.config) as s:
        s.set_integrator("xsph")
        s.rollout_forward(v, MU, sc.dt, T, T)
        ends.append(state(s))
    same(*ends)
