"""The step's sort and cell table at counts around the sort's tiles (512 keys up
to 65,536, 2,048 up to 524,288, then 4,096), from scratch and coherent, several steps in a row (each
leaves the cleared scratch that the next one starts from): the order is the
stable sort of the cell keys, the table its runs.  Whole numbers: equal."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300.solver import ParticleData, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["full", "coherent"])
@pytest.mark.parametrize("n", [1, 31, 511, 512, 513, 4097, 20001, 65536, 65537, 524288, 524289])
def test_step_order_is_the_stable_sort(n, mode):
    sc = scenes.dam_break(1 / 32 if n < 50000 else 1 / 96, (8, 8, 8))
    rng = np.random.default_rng(n)
    x = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    with Solver(ParticleData(x), sc.boundary, sc.config) as s:
        s.debug_sort_mode(mode)
        for _ in range(3):
            before = s.ids()
            f = s.debug_step_fields()
            key_of = np.empty(n, np.uint32)
            key_of[f["ids"]] = f["keys"]
            perm = np.argsort(key_of[before], kind="stable")
            np.testing.assert_array_equal(f["ids"], before[perm])
            np.testing.assert_array_equal(f["keys"], key_of[before][perm])
            _, start = np.unique(f["keys"], return_index=True)
            ranges = np.stack([start, np.append(start[1:], n)], 1)
            used = f["cell_start"] != 0xFFFFFFFF
            got = np.stack([f["cell_start"][used], f["cell_end"][used]], 1)
            np.testing.assert_array_equal(got[np.argsort(got[:, 0])], ranges)
            s.advance(1e-7, 2)
