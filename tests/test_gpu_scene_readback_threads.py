"""Several threads read scenes of one batch at once, each its own and in both
orders: every thread gets its scene, bit for bit.  The scenes take less than one,
one and several of the readback's 4 MiB chunks, read in different orders by the
threads, so that buffers would have to grow under another's read."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import Grid, SolverConfiguration

pytestmark = pytest.mark.gpu

NONE = np.zeros((0, 3), np.float32)
SIZES = [7, 3000, 149796, 149797, 260000, 400000]


@pytest.mark.parametrize("readers", [2, 8])
def test_readers_get_their_scenes(readers):
    rng = np.random.default_rng(readers)
    g = Grid.make_grid((0, 0, 0), (1, 1, 1), 0.01)
    cfg = SolverConfiguration.direct(0.01, 1e-3, 1000.0, 30.0, 5.0, 88.1472, 0.8, g)
    xs = [rng.uniform(0, 1, (n, 3)).astype(np.float32) for n in SIZES]
    vs = [rng.normal(0, 1, (n, 3)).astype(np.float32) for n in SIZES]
    items = [(x, NONE, cfg, v) for x, v in zip(xs, vs)]

    def read(b, first):
        turn = sorted(range(len(SIZES)), key=lambda k: ((k + first) % 3, k))
        return {(k, o): b.scene(k, o) for k in turn for o in ("sorted", "by_id")}

    with Batch(items) as alone, Batch(items) as b, ThreadPoolExecutor(readers) as pool:
        want = read(alone, 0)
        np.testing.assert_array_equal(want[5, "by_id"]["x"], xs[5])
        np.testing.assert_array_equal(want[5, "by_id"]["v"], vs[5])
        for got in pool.map(lambda t: read(b, t), range(3 * readers)):
            for key, fields in want.items():
                for name in fields:
                    np.testing.assert_array_equal(got[key][name], fields[name], err_msg=f"{key} {name}")
