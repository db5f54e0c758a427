"""A batch of few particles in grids of many cells: the cell table is cleared by as many
blocks as it takes, not by one per 256 particles.  A step in 2 x 128^3 cells (33 MB to
clear: 5 us at the memory's rate, about 100 with six blocks) takes at most 50 us more
than one in 2 x 16^3; positions and velocities are the lone solver's bit for bit, from
scratch and coherent."""
import time

import numpy as np
import pytest

from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import Grid, ParticleData, Solver, SolverConfiguration

pytestmark = pytest.mark.gpu

NONE = np.zeros((0, 3), np.float32)


def config(cells):
    g = Grid.make_grid((0, 0, 0), (1, 1, 1), 1 / cells)
    return SolverConfiguration.direct(1 / 128, 1e-3, 1000.0, 30.0, 5.0, 88.1472, 0.8, g)


def test_step_time():
    x = np.random.default_rng(0).uniform(0.2, 0.8, (600, 3)).astype(np.float32)
    per_step = {}
    for cells in (16, 128):
        with Batch([(x, NONE, config(cells))] * 2) as b:
            b.advance(1e-7, 20)
            b.sync()
            best = 1.0
            for _ in range(10):
                t = time.perf_counter()
                b.advance(1e-7, 50)
                b.sync()
                best = min(best, (time.perf_counter() - t) / 50)
            per_step[cells] = best
    assert per_step[128] <= per_step[16] + 50e-6, per_step


@pytest.mark.parametrize("cells", [1, 16, 63, 128])
@pytest.mark.parametrize("sizes", [(1, 600), (0, 257, 5), (3000, 40)])
def test_equal_to_the_solver(sizes, cells):
    rng = np.random.default_rng(cells)
    xs = [rng.uniform(0.3, 0.6, (n, 3)).astype(np.float32) for n in sizes]
    vs = [rng.normal(0, 1, x.shape).astype(np.float32) for x in xs]
    cfg = config(cells)
    with Batch([(x, NONE, cfg, v) for x, v in zip(xs, vs)]) as b:
        b.advance(1e-5, 4)
        for k, (x, v) in enumerate(zip(xs, vs)):
            if not len(x):
                continue
            for mode in ("full", "coherent"):
                with Solver(ParticleData(x), None, cfg, velocities=v) as s:
                    s.debug_sort_mode(mode)
                    s.advance(1e-5, 4)
                    np.testing.assert_array_equal(b.scene(k)["x"], s.positions())
                    np.testing.assert_array_equal(b.scene(k)["v"], s.velocities())
