"""A scene is read back without device memory to pack it in: the readback takes the
neighbour lists', which the next step writes anew."""
import numpy as np
import pytest

from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import Grid, SolverConfiguration
from test_gpu_list_memory import MiB, Short

pytestmark = pytest.mark.gpu

NONE = np.zeros((0, 3), np.float32)


@pytest.mark.parametrize("cap", [96, 16])
def test_read_with_the_memory_full(cap):
    rng = np.random.default_rng(cap)
    g = Grid.make_grid((0, 0, 0), (1, 1, 1), 0.02)
    cfg = SolverConfiguration.direct(0.02, 1e-3, 1000.0, 30.0, 5.0, 88.1472, 0.8, g)
    n = 1 << 20  # 28 MiB to pack
    x = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    v = rng.normal(0, 1, (n, 3)).astype(np.float32)
    items = [(x[:100], NONE, cfg), (x, NONE, cfg, v)]
    with Batch(items) as b, Batch(items) as other:
        for h in (b, other):
            h.debug_list_capacity(cap)
            h.advance(1e-7, 2)
        want = {(k, o): other.scene(k, o) for k in (0, 1) for o in ("sorted", "by_id")}
        b.scene(0)  # the kernel is loaded
        with Short(8 * MiB):
            got = {key: b.scene(*key) for key in want}
            b.advance(1e-7, 2)
            last = b.scene(1)
        other.advance(1e-7, 2)
        for key, fields in want.items():
            for name in fields:
                np.testing.assert_array_equal(got[key][name], fields[name])
        np.testing.assert_array_equal(last["x"], other.scene(1)["x"])
        np.testing.assert_array_equal(last["rho"], other.scene(1)["rho"])
