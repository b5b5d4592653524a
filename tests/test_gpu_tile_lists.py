"""Edges of the particle pass's tiles, lists and windows, of the pair search's cells and of the 2D frame
launch, against the FP64 oracles (GPU tests, through the C ABI).

Tolerances: the device sums FP32 terms, at most N per node. N terms added in any order lie within
N 2^-24 of the exact sum of their magnitudes, and within about sqrt(N) 2^-24 when roundings are independent;
four times that, plus the 1e-6 of a few-particle node used elsewhere, bounds the grid normwise. Positions keep the
1e-6 m of the other step tests, F their 2e-6.
"""
import math

import numpy as np
import pytest

from oracle import oracle as orc
from oracle.oracle2d import Oracle2
from mpm_b200 import scenes
from mpm_b200.params import Domain, Material
from mpm_b200.solver import Solver

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def cloud(n, cells, model=0, seed=3):
    """n particles at random in a cube of `cells` cells that starts on a tile edge of a 16-cell grid."""
    d = scenes.Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=1 / 16, gravity=(0, -9.8, 0), sticky_floor=True)
    rng = np.random.default_rng(seed)
    lo = 4.0 / 16  # node 6 of the grid: base cells from 5.5 on span several tiles
    x = scenes.quantize_positions(lo + rng.uniform(0, cells / 16, (n, 3)), d)
    mat = Material.reference_units(model, E=1e5, density=1000.0) if model in (2, 3) else Material.from_young(model, 1e5, .3)
    sc = scenes._scene("cloud", d, [mat], x, (0, 0, 0))
    sc.m[:] = 1000.0 * (cells / 16) ** 3 / n
    sc.V[:] = (cells / 16) ** 3 / n
    sc.v = np.stack([np.sin(7 * x[:, 1]), np.cos(5 * x[:, 2]), np.sin(6 * x[:, 0])], axis=1)
    return sc


# one particle; a warp, a round of phase A and a scatter round (592), each with one more or less; several
# rounds per tile; 80,000: more than fit the resident CTAs in parts, so whole tiles of about 2,900
@pytest.mark.parametrize("n,cells,model", [(1, 1, 0), (31, 1, 0), (33, 2, 0), (255, 2, 0), (257, 2, 0), (591, 2, 0), (593, 2, 0),
                                           (1300, 2, 0), (2500, 5, 3), (80000, 12, 0)])
def test_tile_counts(n, cells, model):
    sc = cloud(n, cells, model)
    dt = 1e-4
    sol = Solver(sc.domain, n)
    sol.upload(sc)
    st = orc.state_from_scene(sc)
    gm_ref, gp_ref, _ = st.step(dt, want_grid=True)
    tol = 1e-6 + 4 * math.sqrt(27 * n / cells ** 3) * 2.0 ** -24
    gm, gp = sol.grid_debug(dt)
    assert rel(gm, gm_ref) <= tol
    assert rel(gp, gp_ref) <= tol
    sol.step_fixed(dt, 4)
    for _ in range(3):
        st.step(dt)
    out = sol.download(("x", "F"))
    assert np.max(np.abs(out["x"] - st.x)) <= 1e-6
    assert np.max(np.abs(out["F"] - st.F)) <= 2e-6
    assert sol.status() == 0
    sol.close()


# cells travelled per substep: lists kept for the whole run, sorted now and then, sorted every other substep
@pytest.mark.parametrize("cells_per_step", [.0004, .02, .3])
def test_lists_follow_a_moving_body(cells_per_step):
    d = Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=1 / 32)
    mat = Material.from_young(0, 1e5, .3, density=1000.0)
    x = scenes.block_particles(d, (6, 6, 6), (13, 11, 12), 5)
    dt, steps = 1e-4, 40
    v = cells_per_step * d.H / dt
    sc = scenes._scene("moving", d, [mat], x, (v, .7 * v, .4 * v))
    c = x.mean(axis=0)
    sc.v = sc.v + .05 * v * np.stack([x[:, 1] - c[1], c[0] - x[:, 0], 0 * x[:, 2]], axis=1) / d.H / 8
    sol = Solver(sc.domain, sc.n)
    sol.upload(sc)
    st = orc.state_from_scene(sc)
    sol.step_fixed(dt, steps)
    for _ in range(steps):
        st.step(dt)
    out = sol.download(("x", "F"))
    # a position is rounded to H / 2^22 each substep, and each substep adds dt v with FP32's v
    tol = 1e-6 + steps * d.H / 2 ** 23 + 4 * steps * dt * v * 2.0 ** -24
    assert np.max(np.abs(out["x"] - st.x)) <= tol
    assert np.max(np.abs(out["F"] - st.F)) <= 2e-6 * max(1.0, 40 * cells_per_step)
    assert sol.status() == 0
    sol.close()


# the fine cells of a filled grid and the coarse ones of a mostly empty grid
@pytest.mark.parametrize("spacing,radius", [(2.8, 8.0), (.45, .8)])
def test_pair_cells(spacing, radius):
    d = Domain(lower=(-64, -48, -64), upper=(64, 72, 64), H=8.0)
    rng = np.random.default_rng(9)
    n = 1200
    x = rng.uniform(-4 * spacing, 4 * spacing, (n, 3))
    mats = [Material(model=0, mu=.4, lam=.4, specific_heat=cp, conductivity=k) for cp, k in ((4180.0, .6), (450.0, 80.0))]
    sc = scenes._scene("pairs", d, mats, x, (0, 0, 0))
    sc.m, sc.V = rng.uniform(.5, 2.0, n), rng.uniform(.5, 1.5, n)
    sc.mat = (rng.uniform(0, 1, n) < .4).astype(np.int32)
    sc.T = rng.uniform(20, 300, n)
    kw = dict(spacing=spacing, volume_unit=1.0, max_speed=8.0, rate=40.0)
    sol = Solver(d, n)
    sol.upload(sc)
    st = orc.state_from_scene(sc)
    st.init_enthalpy()
    sol.exchange_heat(1 / 60, radius)
    st.exchange_heat(1 / 60, radius=radius)
    assert np.max(np.abs(sol.download(("T",))["T"] - st.T)) <= 1e-4 * 300
    sol.set_regularizer(True, **kw)
    sol.regularize(1 / 240)
    st.regularize(1 / 240, **kw)
    # one rounding of a position to H / 2^22, and FP32 shifts of at most max_speed dt
    assert np.max(np.abs(sol.download(("x",))["x"] - st.x)) <= d.H / 2 ** 22 + 8 / 240 * 4e-6
    sol.close()


# one launch for the frame (one particle per resident thread) and, above that, launches per substep
@pytest.mark.parametrize("nx,ny", [(1, 1), (127, 1), (43, 3), (200, 200)])
def test_plane_frame_launches(nx, ny):
    from mpm_b200.solid_mpm import SolidMPM, SolidSim
    n = nx * ny

    def sim():
        s = SolidSim(n, gravity="center")
        g = np.random.default_rng(4)
        s.count = n
        s.x[:n] = (np.tile(np.arange(nx), ny) - nx / 2) * 3.6 + g.uniform(-.3, .3, n)
        s.y[:n] = (np.repeat(np.arange(ny), nx) - ny / 2) * 3.6 + g.uniform(-.3, .3, n)
        s.vx[:n], s.vy[:n] = g.uniform(-5, 5, n), g.uniform(-5, 5, n)
        s.mass[:n], s.volume[:n], s.material[:n] = 1.1, 1.0, 11
        s.pinned[:n] = g.uniform(0, 1, n) < .02
        s.material[:n][g.uniform(0, 1, n) < .03] = 0  # not a solid: left alone
        return s

    s, t = sim(), sim()
    m, o = SolidMPM(n), Oracle2(n)
    for _ in range(3):
        ng, ag = m.frame(s)
        nc, ac = o.frame(t)
        assert ng == nc and abs(ag - ac) < 1e-9
    extent = 1192.0
    assert np.abs(s.x[:n].astype(np.float64) - t.x[:n]).max() <= 1e-5 * extent
    assert np.abs(s.y[:n].astype(np.float64) - t.y[:n]).max() <= 1e-5 * extent
    assert m.stats(s)["nodes"] == o.stats(t)["nodes"]
    m.close()


# MPM_STATUS_SCATTER_OVERFLOW (0x10) follows from a particle's own tile before and after a move, not from the tile whose
# list holds it. One flyer beside 64 pinned particles (so one stray in 65 keeps the lists); start in cells from the
# grid's origin, velocity in cells, acceleration, substep lengths. In turn: out of a kept list's tile by the near
# side and back across both its sides; out by the far side and on inside the next tile; moves of more than a cell in fresh
# lists that leave the window and that do not; from outside the box into it
@pytest.mark.parametrize("x0,cells,gravity,dts", [(4.51, -.02, True, (1e-4, 1e-2)), (8.49, .02, False, (1e-4, 65e-4)), (7.2, 1.5, False, (1e-4,)),
                                                  (4.6, 2.3, False, (1e-4,)), (7.2, -1.3, False, (1e-4,)), (19.9, -.01, False, (1e-4, 1e-4)),
                                                  (.2, .01, False, (1e-4, 1e-4))])
def test_overflow_status_follows_a_particles_own_tile(x0, cells, gravity, dts):
    h = 1 / 16
    v = cells * h / dts[0]
    g = (1.3 * h / dts[1] - v) / (dts[0] + dts[1]) if gravity else 0.0
    d = Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=h, gravity=(g, 0, 0))
    o = np.asarray(d.origin)
    grid = np.stack(np.meshgrid(*[13.25 + .5 * np.arange(4)] * 3), axis=-1).reshape(-1, 3)
    x = scenes.quantize_positions(o + h * np.concatenate([[[x0, 6.3, 6.3]], grid]), d)
    sc = scenes._scene("flyer", d, [Material.from_young(0, 1e5, .3, density=1000.0)], x, (0, 0, 0))
    sc.v[0, 0] = v
    sc.pinned = (np.arange(len(x)) > 0).astype(np.uint8)
    sol = Solver(d, len(x))
    sol.upload(sc)
    base = lambda p: np.clip(np.floor((p - o) / h - .5), 0, np.asarray(d.dims) - 3).astype(int)
    before, expected = base(x[0]), 0
    for dt in dts:
        sol.step_fixed(dt, 1)
        after = base(sol.download(("x",))["x"][0])
        local = after - (before // 4 * 4 - 1)
        expected |= 0x10 if np.any((local < 0) | (local > 5)) else 0
        assert sol.status() == expected, (before, after)
        before = after
    sol.close()


# around and past half a cell per substep, where two substeps outrun the windows of one list, and past a whole cell
@pytest.mark.parametrize("cells_per_step", [.49, .51, .95, 1.6])
def test_lists_follow_a_fast_body(cells_per_step):
    d = Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=1 / 32)
    mat = Material.from_young(0, 1e5, .3, density=1000.0)
    x = scenes.block_particles(d, (2, 2, 2), (9, 7, 8), 5)
    dt, steps = 1e-5, 12
    v = cells_per_step * d.H / dt
    sc = scenes._scene("fast", d, [mat], x, (v, .7 * v, .4 * v))
    sol = Solver(sc.domain, sc.n)
    sol.upload(sc)
    st = orc.state_from_scene(sc)
    for k in (1, 4, 7):  # the first substep after a fresh scatter, and kept lists between calls
        sol.step_fixed(dt, k)
        for _ in range(k):
            st.step(dt)
    out = sol.download(("x", "F"))
    # as for the slower body: a position is rounded to H / 2^22 each substep, each substep adds dt v with FP32's v
    assert np.max(np.abs(out["x"] - st.x)) <= 1e-6 + steps * d.H / 2 ** 23 + 4 * steps * dt * v * 2.0 ** -24
    assert np.max(np.abs(out["F"] - st.F)) <= 2e-6 * 40 * cells_per_step
    assert sol.status() == (0x10 if cells_per_step > 1 else 0)
    sol.close()


def test_a_fast_body_keeps_to_the_windows():
    """Particles out of the windows are scattered one by one in global memory, at several times the cost of the
    pass: a body at .9 cells per substep takes about the time of one at .3, not more than twice it."""
    d = Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=1 / 128)
    x = scenes.block_particles(d, (3, 3, 3), (67, 19, 35), 5)
    sc = scenes._scene("fast", d, [Material.from_young(0, 1e5, .3, density=1000.0)], x, (0, 0, 0))
    dt, took = 1e-6, {}
    for cells in (.3, .9):
        sc.v[:] = np.array([1, .7, .4]) * cells * d.H / dt
        sol = Solver(d, sc.n)
        sol.upload(sc)
        sol.snapshot()
        sol.profile()
        times = []
        for _ in range(4):
            sol.rollback()
            sol.step_fixed(dt, 1)
            sol.profile_read()
            sol.step_fixed(dt, 20)
            ms, count = sol.profile_read()["g2p2g"]
            times.append(ms / count)
        took[cells] = min(times)
        sol.close()
    assert took[.9] <= 2 * took[.3], took


# the scan of the tile counts over one, two and ten CTAs, with bodies that a run sorts again and again
@pytest.mark.parametrize("grid", [32, 64, 128])
@pytest.mark.parametrize("cells_per_step", [.05, .7])
def test_lists_follow_a_body_on_grids_of_many_tiles(grid, cells_per_step):
    d = Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=1 / grid)
    corner = grid - 26
    x = np.concatenate([scenes.block_particles(d, (2, 2, 2), (9, 7, 8), 5), scenes.block_particles(d, (corner,) * 3, (corner + 5,) * 3, 6)])
    dt, steps = 1e-5, 16
    v = cells_per_step * d.H / dt
    sc = scenes._scene("two bodies", d, [Material.from_young(0, 1e5, .3, density=1000.0)], x, (v, .7 * v, .4 * v))
    sol = Solver(sc.domain, sc.n)
    sol.upload(sc)
    st = orc.state_from_scene(sc)
    sol.step_fixed(dt, steps)
    for _ in range(steps):
        st.step(dt)
    out = sol.download(("x", "F"))
    # as above: positions rounded to H / 2^22, dt v with FP32's v each substep
    assert np.max(np.abs(out["x"] - st.x)) <= 1e-6 + steps * d.H / 2 ** 23 + 4 * steps * dt * v * 2.0 ** -24
    assert np.max(np.abs(out["F"] - st.F)) <= 2e-6 * 40 * cells_per_step
    assert sol.status() == 0
    sol.close()


def test_pair_cells_follow_the_particle_count():
    """One handle with few, many and few particles again: the neighbour cells are the coarse ones, the fine ones and
    the coarse ones of a grid with 1.5 million (regularisation) and 4.9 million (heat exchange) fine cells."""
    d = Domain(lower=(-64, -48, -64), upper=(64, 72, 64), H=8.0)
    mats = [Material(model=0, mu=.4, lam=.4, specific_heat=cp, conductivity=k) for cp, k in ((4180.0, .6), (450.0, 80.0))]
    spacing, radius = 1.39, 1.9
    kw = dict(spacing=spacing, volume_unit=1.0, max_speed=8.0, rate=40.0)
    sol = Solver(d, 100000)
    for n in (1000, 100000, 1000):
        rng = np.random.default_rng(n)
        x = rng.uniform(-.5, .5, (n, 3)) * 1.1 * n ** (1 / 3)
        sc = scenes._scene("pairs", d, mats, x, (0, 0, 0))
        sc.m, sc.V = rng.uniform(.5, 2.0, n), rng.uniform(.5, 1.5, n)
        sc.mat = (rng.uniform(0, 1, n) < .4).astype(np.int32)
        sc.T = rng.uniform(20, 300, n)
        sol.upload(sc)
        st = orc.state_from_scene(sc)
        st.init_enthalpy()
        sol.exchange_heat(1 / 60, radius)
        st.exchange_heat(1 / 60, radius=radius)
        assert np.max(np.abs(sol.download(("T",))["T"] - st.T)) <= 1e-4 * 300  # as in test_pair_cells
        sol.set_regularizer(True, **kw)
        sol.regularize(1 / 240)
        st.regularize(1 / 240, **kw)
        assert np.max(np.abs(sol.download(("x",))["x"] - st.x)) <= d.H / 2 ** 22 + 8 / 240 * 4e-6
    sol.close()


def test_a_pair_pass_costs_by_its_particles_not_the_capacity():
    import time
    d = Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=1 / 128)
    x = scenes.block_particles(d, (4, 4, 4), (9, 9, 9), 1)
    sc = scenes._scene("small", d, [Material.from_young(0, 1e5, .3, density=1000.0)], x, (0, 0, 0))
    took = {}
    for capacity in (sc.n, 4000000):
        sol = Solver(d, capacity)
        sol.upload(sc)
        sol.set_regularizer(True, spacing=d.H / 2, volume_unit=(d.H / 2) ** 3, max_speed=8.0, rate=40.0)
        times = []
        for _ in range(20):
            t0 = time.perf_counter()
            sol.regularize(1e-6)
            times.append(time.perf_counter() - t0)
        took[capacity] = min(times)
        sol.close()
    assert took[4000000] <= 1.5 * took[sc.n], took


# the kinds of pass beside the plain one, each with lists that particles leave: conduction (which also reads node
# temperatures outside the window), pinned particles in the lists, the window without TMA, a history law, and the
# Newton-gated and learned returns with a body that yields
@pytest.mark.parametrize("kind", ["conduction", "pinned", "plain loads", "sand", "newton", "learned"])
@pytest.mark.parametrize("cells_per_step", [.04, .3, .8])
def test_kept_lists_in_every_kind_of_pass(kind, cells_per_step, monkeypatch):
    d = Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=1 / 32)
    yields = kind in ("newton", "learned")
    dt, steps = 1e-6 if yields else 1e-5, 14
    v = cells_per_step * d.H / dt
    x = scenes.block_particles(d, (3, 3, 3), (10, 8, 9), 5)
    mat = Material.from_young(0, 1e5, .3, density=1000.0, specific_heat=1000.0)
    if yields:
        mat = scenes.johnson_cook_metal(7)
    if kind == "sand":
        mat = Material.reference_units(3, E=1e5, density=1000.0)
    if kind == "pinned":  # a fixed block three cells beside the moving one's path, in the same tiles
        x = np.concatenate([x, scenes.block_particles(d, (3, 3, 13), (12, 8, 15), 6)])
    sc = scenes._scene(kind, d, [mat], x, (v, 0, 0))
    if kind == "pinned":
        sc.pinned = (x[:, 2] > 11 * d.H).astype(np.uint8)
        sc.v[sc.pinned == 1] = 0
    if kind == "conduction":
        sc.T = np.where(x[:, 0] < 6.5 * d.H, 400.0, 300.0)
        sc.meta["conduction"] = dict(k=5e5, rho=1000.0, cp=1000.0)
    if yields:
        sc.F = np.tile((np.eye(3) + np.diag([.008, -.004, -.004])).ravel(), (sc.n, 1))
    if kind == "plain loads":
        monkeypatch.setenv("MPM_B200_NO_TMA", "1")
    sol = Solver(d, sc.n)
    sol.upload(sc)
    if kind == "newton":
        sol.set_return_mode(mode="newton", gate_tol=1e-5, newton=8)
    if kind == "learned":
        from mpm_b200.surrogate import Surrogate
        net = Surrogate(mat, seed=3)
        sol.set_return_mode(net, gate_tol=1e-5, newton=4)
        net.close()
    st = orc.state_from_scene(sc)
    sol.step_fixed(dt, steps)
    for _ in range(steps):
        st.step(dt)
    out = sol.download(("x", "F", "T", "ep"))
    assert sol.status() == 0
    # the bounds of the moving body above; temperatures and plastic strain as in their own tests
    assert np.max(np.abs(out["x"] - st.x)) <= 1e-6 + steps * d.H / 2 ** 23 + 4 * steps * dt * v * 2.0 ** -24
    assert np.max(np.abs(out["F"] - st.F)) <= 2e-6 * max(1.0, 40 * cells_per_step)
    if kind == "conduction":
        assert np.max(np.abs(out["T"] - st.T)) <= 1e-5 * 100
    if yields:
        assert np.max(st.ep) > 0
        assert np.max(np.abs(out["ep"] - st.ep)) <= 2e-6 + 1e-4 * np.max(st.ep)
    sol.close()


# a batch whose one fast scene holds too few of its particles to bring a sort by their share, eagerly and in a graph
@pytest.mark.parametrize("graph", [False, True])
def test_kept_lists_of_a_batch_with_one_fast_scene(graph):
    from mpm_b200.solver import Batch
    subs, steps = [], 72
    for k in range(3):
        d = Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=1 / 48)
        fast = k == 1
        x = scenes.block_particles(d, (3, 3, 3), (5, 5, 5) if fast else (13, 13, 13), 60 + k)
        subs.append(scenes._scene("s%d" % k, d, [Material.from_young(0, 1e5, .3, density=1000.0)], x, (240.0 if fast else .5, 0, 0)))
    b = Batch(subs)
    b.upload()
    b.run(steps, graph=graph)
    parts, times = b.split(b.download(("x", "F"))), b.times()[0]
    assert b.status() == 0
    b.close()
    for k, sc in enumerate(subs):
        st, t = orc.state_from_scene(sc), 0.0
        for _ in range(steps):
            dt = st.stable_dt()
            st.step(dt)
            t += dt
        far = abs(sc.v[0, 0]) * t
        # the time follows from FP32 maxima (four roundings of 2^-24 a substep at most); positions as above
        assert abs(times[k] - t) <= 4 * 2.0 ** -24 * t * steps ** .5 + 1e-6 * t
        assert np.max(np.abs(parts[k]["x"] - st.x)) <= 1e-6 + steps * sc.domain.H / 2 ** 23 + 8 * 2.0 ** -24 * far + 2e-6 * far
        assert np.max(np.abs(parts[k]["F"] - st.F)) <= 2e-6 * 16


# sorts in 24 substeps beside the first scatter's: none while a body stays, at most every other substep while lists last two of
# them, every one past half a cell
@pytest.mark.parametrize("cells_per_step,least,most", [(0.0, 0, 0), (.0004, 0, 0), (.3, 8, 13), (.8, 22, 24)])
def test_sorts_follow_the_motion(cells_per_step, least, most):
    d = Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=1 / 64)
    x = scenes.block_particles(d, (2, 2, 2), (12, 8, 9), 5)
    dt = 1e-6
    sc = scenes._scene("moving", d, [Material.from_young(0, 1e5, .3, density=1000.0)], x, (cells_per_step * d.H / dt, 0, 0))
    sol = Solver(d, sc.n)
    sol.upload(sc)
    sol.step_fixed(dt, 24)
    assert least <= sol.sort_count() - 1 <= most
    sol.close()


# whole tiles and parts on both sides of the rule's lines, of 56,832, 113,664 and 189,440 particles on 148 SMs
@pytest.mark.parametrize("n,model", [(56832, 0), (56833, 0), (113664, 3), (113665, 3), (189441, 3)])
def test_tile_parts_on_both_sides_of_their_lines(n, model):
    test_tile_counts(n, 12, model)
