"""Two-scale steps where lists overflow: coarse particles with more fine neighbours than
320, supports that hold more particles than a same-population list (whose lists then
have 64 entries), and totals on both sides of 2^20 particles, from where on the
coarse particles beside fine ones take one lane in the density pass.  One step from rest
against the FP64 oracle with the bounds of test_gpu_two_scale_lanes."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300.solver import Grid
from sph2s_final_gb300.two_scale import HIGH, LOW, Solver2
from test_gpu_two_scale_lanes import ACC_TOL, CAPACITY, RHO_TOL, oracle

pytestmark = pytest.mark.gpu


def check(low, high, sc):
    """Counts of the lists that fit (64 entries in any case), densities, accelerations."""
    with Solver2(low, high, sc.boundary, sc.config, len(low) + 64, len(high) + 64) as s:
        of = oracle(s, sc).step_fields(sc.dt)
        s.advance(sc.dt, 1)
        overflow = []
        for r in (LOW, HIGH):
            d, st = s.debug_last_step(r), s.state(r)
            np.testing.assert_array_equal(d["ids"], of["ids"][r])
            for got, want, least, most in (
                    (d["nbr_same"], of["nbr_same"][r] - 1, 64, 96),
                    (d["nbr_compl"], of["nbr_compl"][r], CAPACITY[r], CAPACITY[r])):
                np.testing.assert_array_equal(got[want <= least], want[want <= least])
                assert (got[want > most] > most).all()
                assert ((got == want) | (got > most)).all()
                overflow.append(int((want > most).sum()))
            rel = np.abs(d["rho"] - of["rho"][r]) / of["rho"][r]
            assert rel.max() <= RHO_TOL, (r, rel.max())
            acc = st["v"].astype(np.float64) / float(np.float32(sc.dt))
            err = np.abs(acc - of["acc"][r]).max() / np.abs(of["acc"][r]).max()
            assert err <= ACC_TOL, (r, err)
        return overflow


def slab_scene(k, inv, h_over_s, coupled, seed=0):
    """Coarse sites of a k^3 lattice on one side, fine ones on the other, some of them
    among the coarse ones."""
    sc = scenes.two_scale_dam_break(1 / inv, (k, k, k), dt=1e-6, slab=(2.0, 3.0))
    h = float(np.float32(h_over_s * sc.spacing))
    for r, hr in enumerate((h, float(np.float32(0.5) * np.float32(h)))):
        sc.config.effective_radius[r] = hr
        sc.config.grid[r] = Grid.make_grid((0, 0, 0), (1, 1, 1), hr)
    sc.config.mode = 1 if coupled else 0
    x = sc.low.positions
    low = x[x[:, 0] < 0.6 * k * sc.spacing]
    n = k // 2
    fine = scenes.lattice_block(0.5 * sc.spacing, (n, 2 * k, 2 * k))
    fine = fine + np.float32([0.4 * k * sc.spacing, 0, 0])
    return sc, low, scenes.jitter(fine, sc.spacing, 0.005, seed)


@pytest.mark.parametrize("coupled", [False, True])
@pytest.mark.parametrize("h", [2.0, 2.5, 3.0, 3.5])
@pytest.mark.parametrize("k,inv", [(14, 32), (40, 84)])
def test_supports(k, inv, h, coupled):
    sc, low, high = slab_scene(k, inv, h, coupled)
    assert (len(low) + len(high) < 49152) == (k == 14)
    overflow = check(low, high, sc)
    assert (overflow[1] > 0) == (h >= 2.5)  # coarse particles' fine neighbours
    assert (overflow[0] > 0 and overflow[2] > 0) == (h >= 3.0)  # each population's own


@pytest.mark.parametrize("total", [(1 << 20) - 1, 1 << 20])
def test_sizes_at_which_the_near_density_changes(total):
    sc = scenes.two_scale_dam_break(1 / 200, (110, 100, 100), dt=1e-6, slab=(2.0, 3.0), border=1)
    rng = np.random.default_rng(5)
    high = rng.uniform(0.1, 0.3, (20000, 3)).astype(np.float32)
    low = sc.low.positions[:total - len(high)]
    assert len(low) + len(high) == total
    check(low, high, sc)
