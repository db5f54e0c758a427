"""Gradients of a rollout where particles have more neighbours than a list holds (96
entries), so that the adjoint passes find them again in the stencil: directional
derivatives against central differences of the FP64 rollout, and the batched rollout
against the single one, bit for bit.

Tolerance as in test_gpu_adjoint_sizes: FP32 roundings of the perturbed velocities
and of the gradients' sums, 1e-3 of the derivative plus 1e-4 of |grad||d|."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300.autograd import node_grid
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import ParticleData, Solver
from test_gpu_adjoint_sizes import EPS, MU, STEPS, loss64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crowd", [97, 98, 130])
@pytest.mark.parametrize("alone", [True, False])
def test_gradients(crowd, alone):
    sc, _ = scenes.differentiable_scene((6, 7, 5))
    rng = np.random.default_rng(crowd)
    h = float(sc.config.effective_radius)
    # a jittered lattice of spacing 0.09 h: every pair within h, none nearly coincident
    side = scenes.lattice_block(1.0, (6, 6, 6))
    side = side[np.argsort(((side - 2.5) ** 2).sum(1), kind="stable")][:crowd] - 2.5
    ball = (np.float32([0.6, 0.6, 0.6]) + (side + rng.uniform(-0.2, 0.2, side.shape)) * 0.09 * h)
    x = ball.astype(np.float32)
    assert np.linalg.norm(x[:, None] - x[None], axis=2).max() < h
    if not alone:
        x = np.concatenate([sc.fluid.positions, x])
    sc.dt = 1e-5
    v = rng.normal(0, 0.1, x.shape).astype(np.float32)
    target = rng.uniform(0, 800, 32 ** 3).astype(np.float32)
    with Solver(ParticleData(x), sc.boundary, sc.config) as s:
        s.rollout_forward(v, MU, sc.dt, STEPS, 2)
        s.rollout_density_loss(node_grid(), target)
        gv, gx, gmu = s.rollout_backward()
        assert s.debug_step_fields()["nbr_fluid"].max() == crowd  # itself included
    g = gv.astype(np.float64)
    scale = np.linalg.norm(v)
    for d in (g, rng.normal(size=v.shape)):
        d = d * (scale / np.linalg.norm(d))
        fd = (loss64(sc, x, v + EPS * d, target) - loss64(sc, x, v - EPS * d, target)) / (2 * EPS)
        assert abs((g * d).sum() - fd) <= 1e-3 * abs(fd) + 1e-4 * np.linalg.norm(g) * scale
    sc.config.viscosity = MU
    with Batch([(x, sc.boundary.positions, sc.config)] * 2) as b:
        b.rollout_forward([v, v], np.full(2, MU, np.float32), sc.dt, STEPS, 2)
        b.rollout_density_loss([node_grid()] * 2, [target] * 2)
        bv, bx, bmu = b.rollout_backward()
    for k in range(2):
        np.testing.assert_array_equal(bv[k], gv)
        np.testing.assert_array_equal(bx[k], gx)
        assert bmu[k] == gmu
