"""Neighbour lists have 96 entries, or fewer where the device memory does not hold
them.  Every capacity gives the same results (a particle with more neighbours than
its list holds finds them again): the steps of the solver, of XSPH, of a batch and
the rollout's gradients bit for bit, the two-scale step within the rounding of its
sums' order.  With the memory short, handles and tapes that fit with lists of 64
entries and less are created and run."""
import numpy as np
import pytest

from sph2s_final_gb300 import scenes
from sph2s_final_gb300._abi import SphError
from sph2s_final_gb300.autograd import node_grid
from sph2s_final_gb300.batched import Batch
from sph2s_final_gb300.solver import Grid, ParticleData, Solver, SolverConfiguration
from sph2s_final_gb300.two_scale import HIGH, LOW, Solver2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CAPS = [4, 16, 32, 36, 48, 64, 92]
MU = 3.0


def single(sc, v, cap, xsph):
    with Solver(sc.fluid, sc.boundary, sc.config, velocities=v) as s:
        if cap:
            s.debug_list_capacity(cap)
        if xsph:
            s.set_integrator("xsph")
        s.advance(sc.dt, 3)
        return s.positions(), s.velocities(), s.densities()


@pytest.mark.parametrize("xsph", [False, True])
@pytest.mark.parametrize("side", [12, 26])  # nine lanes to a particle in the density pass, and one
def test_solver_steps(side, xsph):
    sc, v = scenes.differentiable_scene((side, side, side))
    sc.config.xsph_coeff = 0.3
    want = single(sc, v, None, xsph)
    for cap in CAPS:
        for a, b in zip(single(sc, v, cap, xsph), want):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("cap", CAPS)
def test_batch_and_gradients(cap):
    sc, v = scenes.differentiable_scene((9, 13, 11))
    sc.config.viscosity = MU
    target = np.random.default_rng(3).uniform(0, 800, 32 ** 3).astype(np.float32)
    items = [(sc.fluid.positions, sc.boundary.positions, sc.config)] * 2
    with Solver(sc.fluid, sc.boundary, sc.config) as s, \
            Solver(sc.fluid, sc.boundary, sc.config) as t, Batch(items) as b:
        t.debug_list_capacity(cap)
        b.debug_list_capacity(cap)
        for r in (s, t):
            r.rollout_forward(v, MU, sc.dt, 5, 2)
            r.rollout_density_loss(node_grid(), target)
        want, got = s.rollout_backward(), t.rollout_backward()
        for a, w in zip(got, want):
            np.testing.assert_array_equal(np.asarray(a), np.asarray(w))
        b.rollout_forward([v, v], np.full(2, MU, np.float32), sc.dt, 5, 2)
        np.testing.assert_array_equal(b.scene(1)["x"], scene_end(sc, v, 5))
        b.rollout_density_loss([node_grid()] * 2, [target] * 2)
        gv, gx, gmu = b.rollout_backward()
        for k in range(2):
            np.testing.assert_array_equal(gv[k], want[0])
            np.testing.assert_array_equal(gx[k], want[1])
            assert gmu[k] == want[2]


def scene_end(sc, v, steps):
    with Solver(sc.fluid, sc.boundary, sc.config, velocities=v) as s:
        s.advance(sc.dt, steps)
        return s.positions()


@pytest.mark.parametrize("big", [False, True])
def test_two_scale_step(big):
    """Both sides of the size that decides between several lanes for every particle
    and for the coarse ones beside fine ones alone.  The sums' order differs, each of
    ~300 terms: 300 roundings of 6e-8, 2e-5 of the largest acceleration."""
    k = 40 if big else 12
    sc = scenes.two_scale_dam_break(1 / 80 if big else 1 / 32, (k, k, 32 if big else k), dt=1e-5,
                                    slab=(2.0, 3.0))
    high = np.random.default_rng(1).uniform(0.05, 0.2, (3000, 3)).astype(np.float32)
    assert (len(sc.low.positions) + len(high) >= 49152) == big

    def step(cap):
        with Solver2(sc.low, high, sc.boundary, sc.config) as s:
            if cap:
                s.debug_list_capacity(cap)
            s.advance(sc.dt, 1)
            return [s.state(r)["v"] / sc.dt for r in (LOW, HIGH)]

    want = step(None)
    for cap in (4, 32, 64):
        for a, w in zip(step(cap), want):
            assert np.abs(a - w).max() <= 2e-5 * np.abs(w).max()


@pytest.mark.parametrize("entries", [0, 2, 6, 97, 100])
def test_capacity_refused(entries):
    sc = scenes.small_scene(5)
    with Solver(sc.fluid, sc.boundary, sc.config) as s:
        with pytest.raises(SphError, match="SPH_E_INVALID"):
            s.debug_list_capacity(entries)


class Short:
    """Device memory with `left` bytes free."""

    def __init__(self, left):
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.held = torch.empty(max(0, free - left), dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        del self.held
        torch.cuda.empty_cache()


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


N = 1 << 20


@pytest.fixture(scope="module")
def cloud():
    rng = np.random.default_rng(4)
    g = Grid.make_grid((0, 0, 0), (1, 1, 1), 0.02)
    cfg = SolverConfiguration.direct(0.02, 1e-3, 1000.0, 30.0, MU, 88.1472, 0.8, g)
    x = scenes.jitter(scenes.lattice_block(0.01, (100, 100, 105))[:N], 0.01, 0.01, 2)
    return x, rng.normal(0, 0.1, x.shape).astype(np.float32), cfg


MiB = 1 << 20


@pytest.mark.parametrize("short", [64, 168, 232, 296])
def test_handles_when_memory_is_short(cloud, short):
    """The lists of 1,048,576 particles: 384 MiB with 96 entries; 64, 48, 32 and 16
    entries are 128, 192, 256 and 320 MiB less."""
    x, v, cfg = cloud
    none = np.zeros((0, 3), np.float32)
    with Solver(ParticleData(x), None, cfg, velocities=v) as s, \
            Batch([(x, none, cfg, v), (x[:7], none, cfg)]) as b:  # the kernels are loaded
        s.advance(1e-5, 2)
        b.advance(1e-5, 2)
        want = s.positions(), s.velocities()
        b.sync()
    for make, read in ((lambda: Solver(ParticleData(x), None, cfg, velocities=v),
                        lambda h: (h.positions(), h.velocities())),
                       (lambda: Batch([(x, none, cfg, v), (x[:7], none, cfg)]),
                        lambda h: (h.scene(0)["x"], h.scene(0)["v"]))):
        before = free_bytes()
        with make():
            used = before - free_bytes()
        with Short(used - short * MiB + 24 * MiB):
            h = make()
            h.advance(1e-5, 2)
            h.sync()
        with h:
            for a, w in zip(read(h), want):
                np.testing.assert_array_equal(a, w)


@pytest.mark.parametrize("short", [128, 512])
def test_tape_when_memory_is_short(cloud, short):
    x, v, cfg = cloud
    target = np.zeros(16 ** 3, np.float32)

    def run(s):
        s.rollout_density_loss(node_grid((16, 16, 16)), target)
        return s.rollout_backward()

    with Solver(ParticleData(x), None, cfg) as s:
        before = free_bytes()
        s.rollout_forward(v, MU, 1e-5, 2, 2)
        used = before - free_bytes()
        want = run(s)
    with Solver(ParticleData(x), None, cfg) as s:
        s.advance(1e-5, 1)
        s.sync()
        with Short(used - short * MiB + 24 * MiB):
            s.rollout_forward(v, MU, 1e-5, 2, 2)
        for a, w in zip(run(s), want):
            np.testing.assert_array_equal(np.asarray(a), np.asarray(w))


def test_lists_beyond_a_quarter_of_the_memory():
    """4,200,000 particles' lists: 1,538 MiB with 96 entries, 1,025 with 64, which they
    have where less than four times the former is free."""
    n = 4200000
    g = Grid.make_grid((0, 0, 0), (1, 1, 1), 0.02)
    cfg = SolverConfiguration.direct(0.02, 1e-3, 1000.0, 30.0, MU, 88.1472, 0.8, g)
    x = scenes.jitter(scenes.lattice_block(1 / 170, (162, 162, 162))[:n], 1 / 170, 0.01, 2)

    def make():
        before = free_bytes()
        s = Solver(ParticleData(x), None, cfg)
        return s, before - free_bytes()

    s, much = make()
    with s:
        s.advance(1e-6, 2)
        want = s.positions()
    with Short(6000 * MiB):
        s, less = make()
        with s:
            s.advance(1e-6, 2)
            np.testing.assert_array_equal(s.positions(), want)
    assert abs((much - less) - 4 * 32 * n) <= 16 * MiB
