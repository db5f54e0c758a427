"""Coarse particles beside fine ones take passes of their own, several lanes to
a particle: one step against the oracle (the bounds of test_gpu_two_scale) where
that can go wrong: a single neighbour, counts around the lanes, fine particles
in one row of cells (one lane's share overflows, the list does not), a ball with
more fine particles than a list holds, populations that appear later, and steps
far enough on to run as an updated graph.  Small scenes (below 49,152 particles)
give every particle several lanes; one larger scene has them near alone."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300.two_scale import Solver2
from test_gpu_two_scale import check_step

pytestmark = pytest.mark.gpu


def scene(coupled, slab=(2.0, 3.0)):
    sc = scenes.two_scale_dam_break(1 / 32, (12, 9, 7), dt=2e-5, slab=slab)
    sc.config.mode = 1 if coupled else 0
    return sc


def fine(kind, rng):
    centre = np.float32([0.21, 0.17, 0.12])
    if kind == "one":
        return centre[None]
    if kind == "ragged":
        return rng.uniform(0.05, 0.3, (1001, 3))
    if kind == "row":  # along x, within one row of fine cells
        return centre + np.stack([np.linspace(-0.04, 0.04, 150), rng.uniform(0, 0.004, 150),
                                  rng.uniform(0, 0.004, 150)], 1)
    return centre + rng.uniform(-0.025, 0.025, (700, 3))  # "ball"


@pytest.mark.parametrize("coupled", [False, True])
@pytest.mark.parametrize("kind", ["one", "ragged", "row", "ball"])
def test_near_particles(kind, coupled):
    sc = scene(coupled)
    high = fine(kind, np.random.default_rng(6)).astype(np.float32)
    for low in (sc.low.positions, sc.low.positions[:1], sc.low.positions[:33]):
        with Solver2(low, high, sc.boundary, sc.config) as s:
            check_step(s, sc)


@pytest.mark.parametrize("coupled", [False, True])
@pytest.mark.parametrize("kind", ["one", "ragged", "row", "ball"])
def test_near_particles_of_a_larger_scene(kind, coupled):
    sc = scenes.two_scale_dam_break(1 / 80, (40, 36, 36), dt=8e-6, slab=(2.0, 3.0))
    sc.config.mode = 1 if coupled else 0
    high = (0.4 * fine(kind, np.random.default_rng(6))).astype(np.float32)
    assert len(sc.low.positions) >= 49152
    with Solver2(sc.low.positions, high, sc.boundary, sc.config) as s:
        check_step(s, sc)


def test_sizes_that_change_while_the_step_is_a_graph():
    """No fine particles at first, then splits on most steps: the step's graph is
    made, updated and remade when nodes come and go."""
    sc = scenes.two_scale_dam_break(1 / 32, (12, 9, 7), dt=5e-4, slab=(0.36, 0.64))
    x = sc.low.positions + np.float32([-0.0005, 0.05, 0.05])
    with Solver2(x, None, sc.boundary, sc.config) as s:
        seen = set()
        for k in range(40):
            s.advance(sc.dt, 3)
            check_step(s, sc)
            seen.add(tuple(s.counts().values()))
        assert len(seen) > 3
