"""The rollout's backward pass at particle counts around the widths its kernels
work in (8 lanes to a particle near the boundary, 32 to a warp, 256 to a block,
blocks summed by 32 lanes), inside the box and with particles beyond its wall:
directional derivatives against central differences of the FP64 rollout, and
the batched rollout against the single one, bit for bit.

Tolerance: the perturbed velocities are rounded to FP32 (6e-8 of |v| against a
step of 1e-3 of it, so 6e-5 of |grad||d|) and the gradients are FP32 sums (about
1e-5 of their terms): 1e-3 of the derivative plus 1e-4 of |grad||d|."""
import numpy as np
import pytest

from oracle import oracle as O
from sph2s_final_gb300 import scenes
from sph2s_final_gb300.autograd import node_grid
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import ParticleData, Solver

pytestmark = pytest.mark.gpu

STEPS, MU, EPS = 3, 3.0, 1e-3


def loss64(sc, x, v, target):
    cfg = sc.config
    old, cfg.viscosity = cfg.viscosity, MU
    ro = O.SSRollout(cfg, x, sc.boundary.positions, v)
    ro.advance(sc.dt, STEPS)
    cfg.viscosity = old
    return O.splat_loss(cfg, ro.state()["x"], target=target)[1]


@pytest.mark.parametrize("lattice,shift", [
    ((1, 1, 1), 0.0), ((3, 3, 1), 0.0), ((11, 3, 1), 0.0), ((8, 8, 4), 0.0), ((43, 2, 3), 0.0),
    ((5, 6, 7), -0.02), ((21, 20, 20), 0.0)])
def test_gradients_at_ragged_counts(lattice, shift):
    sc, v = scenes.differentiable_scene(lattice)
    x = (sc.fluid.positions + np.float32([shift, 0, 0])).astype(np.float32)
    rng = np.random.default_rng(7)
    target = rng.uniform(0, 800, 32 ** 3).astype(np.float32)
    with Solver(ParticleData(x), sc.boundary, sc.config) as s:
        s.rollout_forward(v, MU, sc.dt, STEPS, 2)
        s.rollout_density_loss(node_grid(), target)
        gv, gx, gmu = s.rollout_backward()
    g = gv.astype(np.float64)
    scale = np.linalg.norm(v)
    for d in (g, rng.normal(size=v.shape)):
        d = d * (scale / np.linalg.norm(d))
        fd = (loss64(sc, x, v + EPS * d, target) - loss64(sc, x, v - EPS * d, target)) / (2 * EPS)
        assert abs((g * d).sum() - fd) <= 1e-3 * abs(fd) + 1e-4 * np.linalg.norm(g) * scale
    old, sc.config.viscosity = sc.config.viscosity, MU
    with Batch([(x, sc.boundary.positions, sc.config)] * 2) as b:
        b.rollout_forward([v, v], np.full(2, MU, np.float32), sc.dt, STEPS, 2)
        b.rollout_density_loss([node_grid()] * 2, [target] * 2)
        bv, bx, bmu = b.rollout_backward()
    sc.config.viscosity = old
    for k in range(2):
        np.testing.assert_array_equal(bv[k], gv)
        np.testing.assert_array_equal(bx[k], gx)
        assert bmu[k] == gmu
