"""The two-scale kernels that a step runs: several lanes to every particle below
49,152 of them, from there on to the coarse particles beside fine ones.  One step
from rest against the FP64 oracle, densities and list lengths as the step left them
and accelerations as v' / dt: neighbour counts bit-exact, densities <= 1e-5 relative
per particle, accelerations <= 1e-5 max-norm relative (v' = fma(dt, a, 0) rounds a by
another 6e-8).  Colours and the surface trigger in a scene that takes both kinds of
kernel."""
import numpy as np
import pytest

from oracle.oracle_ts import TSRollout
from sph2s_final_gb300 import scenes
from sph2s_final_gb300.two_scale import HIGH, LOW, Solver2
from test_gpu_two_scale_near import fine

pytestmark = pytest.mark.gpu

RHO_TOL = ACC_TOL = 1e-5
CAPACITY = {LOW: 320, HIGH: 64}  # complementary lists
SMALL = 49152  # kTsSmall


def oracle(s, sc):
    nl, nh = s.next_ids()
    return TSRollout(sc.config, sc.boundary.positions, [s.state(LOW), s.state(HIGH)],
                     group_base=s.counts()["groups"], pid_base=[nl, nh])


def check_from_rest(low, high, sc):
    with Solver2(low, high, sc.boundary, sc.config) as s:
        of = oracle(s, sc).step_fields(sc.dt)
        s.advance(sc.dt, 1)
        for r in (LOW, HIGH):
            d, st = s.debug_last_step(r), s.state(r)
            np.testing.assert_array_equal(d["ids"], of["ids"][r])
            np.testing.assert_array_equal(st["ids"], of["ids"][r])
            if not d["ids"].size:
                continue
            for got, want, most in ((d["nbr_same"], of["nbr_same"][r] - 1, 96),
                                    (d["nbr_compl"], of["nbr_compl"][r], CAPACITY[r])):
                fits = want <= most
                np.testing.assert_array_equal(got[fits], want[fits])
                assert (got[~fits] > most).all()
            rel = np.abs(d["rho"] - of["rho"][r]) / of["rho"][r]
            assert rel.max() <= RHO_TOL, (r, rel.max())
            acc = st["v"].astype(np.float64) / float(np.float32(sc.dt))
            err = np.abs(acc - of["acc"][r]).max() / np.abs(of["acc"][r]).max()
            assert err <= ACC_TOL, (r, err)


@pytest.mark.parametrize("coupled", [False, True])
@pytest.mark.parametrize("kind", ["one", "ragged", "row", "ball"])
def test_small_scene(kind, coupled):
    sc = scenes.two_scale_dam_break(1 / 32, (12, 9, 7), dt=1e-6, slab=(2.0, 3.0))
    sc.config.mode = 1 if coupled else 0
    high = fine(kind, np.random.default_rng(6)).astype(np.float32)
    for low in (sc.low.positions, sc.low.positions[:1], sc.low.positions[:33],
                np.zeros((0, 3), np.float32)):
        check_from_rest(low, high, sc)
    check_from_rest(sc.low.positions, None, sc)


@pytest.mark.parametrize("coupled", [False, True])
@pytest.mark.parametrize("kind,total", [("one", None), ("ragged", SMALL - 1), ("ragged", SMALL),
                                        ("ragged", None), ("row", None), ("ball", None)])
def test_larger_scene(kind, total, coupled):
    sc = scenes.two_scale_dam_break(1 / 80, (40, 36, 36), dt=1e-6, slab=(2.0, 3.0))
    sc.config.mode = 1 if coupled else 0
    high = (0.4 * fine(kind, np.random.default_rng(6))).astype(np.float32)
    low = sc.low.positions if total is None else sc.low.positions[:total - len(high)]
    check_from_rest(low, high, sc)


def large(surface):
    sc = scenes.two_scale_dam_break(1 / 80, (40, 36, 36), dt=1e-4,
                                    slab=(2.0, 3.0), blend_increment=0.25)
    if surface:
        sc.config.split_trigger = 1  # SPH2_SPLIT_SURFACE
        sc.config.surface_density = 1.0
    high = np.random.default_rng(6).uniform(0.02, 0.3, (20000, 3)).astype(np.float32)
    return sc, high


def test_colours_of_a_larger_scene():
    sc, high = large(False)
    with Solver2(sc.low.positions, high, sc.boundary, sc.config) as s:
        s.set_color_output(True)
        s.advance(sc.dt, 3)
        of = oracle(s, sc).step_fields(sc.dt)
        s.advance(sc.dt, 1)
        for r in (LOW, HIGH):
            col, ids = s.colors(r)
            np.testing.assert_array_equal(ids, of["ids"][r])
            ok = np.abs(of["dist_cm"][r] - 0.0025) > 1e-6
            assert ok.mean() > 0.99
            assert np.abs(col[ok] - of["colour"][r][ok]).max() <= 1e-4


def test_surface_trigger_of_a_larger_scene():
    """The trigger density lies in the widest gap between the coarse particles' own
    densities between 700 and 1,000, so rounding decides nothing at the first step; later ones
    may differ by as many particles as have a density within 1e-5 of it."""
    sc, high = large(True)
    with Solver2(sc.low.positions, high, sc.boundary, sc.config) as s:
        rho = np.sort(oracle(s, sc).step_fields(sc.dt)["rho"][LOW])
    near = rho[(rho > 700) & (rho < 1000)]
    k = np.argmax(np.diff(near))
    trigger = np.float32(0.5 * (near[k] + near[k + 1]))
    assert near[k + 1] - near[k] > 4e-5 * trigger
    sc.config.surface_density = float(trigger)
    with Solver2(sc.low.positions, high, sc.boundary, sc.config) as s:
        splits = 0
        for step in range(3):
            ro = oracle(s, sc)
            of = ro.step_fields(sc.dt)
            close = sum(int((np.abs(of["rho"][r] / trigger - 1) < 1e-5).sum()) for r in (LOW, HIGH))
            assert step > 0 or not (np.abs(of["rho"][LOW] / trigger - 1) < 1e-5).any()
            s.advance(sc.dt, 1)
            got, want = s.last_stats(), ro.last_stats()
            for key in want:
                assert abs(got[key] - want[key]) <= (close if step else 0), (step, key)
            splits += got["splits"]
            if got != want:
                break
        assert splits > 100
