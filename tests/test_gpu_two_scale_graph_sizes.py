"""A scene that grows past 49,152 particles by splits while its step runs as a graph: the
step's kernels are others from there on, and the graph is updated or made anew.  Every
third step against the oracle (the bounds of test_gpu_two_scale)."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300.two_scale import Solver2
from test_gpu_two_scale import check_step

pytestmark = pytest.mark.gpu


def test_growth_past_the_small_scene():
    sc = scenes.two_scale_dam_break(1 / 80, (40, 36, 33), dt=2e-4, slab=(0.4885, 0.8))
    with Solver2(sc.low, None, sc.boundary, sc.config) as s:
        totals = []
        for _ in range(24):
            s.advance(sc.dt, 2)
            check_step(s, sc)
            c = s.counts()
            totals.append(c["low"] + c["high"])
        grown = np.array(totals) >= 49152
        assert not grown[:2].any() and grown[-1], totals
