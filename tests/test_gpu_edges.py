"""Edges of the accepted range, and what stands beside the step: one-point sides, long lines, strong
dispersion, source counts at a tile's limit, reads while another simulation runs, set-up costs, size rules.

Tolerance as in test_gpu_any_length.py: about ten transforms a step, each adding some 2e-7 of relative
rounding error, below 3e-5 over 60 steps.
"""
import threading

import numpy as np
import pytest

from _util import assert_parity, errors, run_gpu, run_oracle
from test_gpu_any_length import TOL_L2, TOL_MAX, check, make_case

pytestmark = pytest.mark.gpu


# a one-point side has the derivative 0 (its only multiplier is k = 0): on the in-place passes alone,
# beside register passes (64, 48 and 96 points), in a volume of one slice, and as a whole 1-D grid
@pytest.mark.parametrize("shape", [(64, 1), (1, 64), (1, 22), (48, 40, 1), (96, 1, 40), (1, 40, 33), (64, 1, 1), (1, 1), (1,)])
@pytest.mark.parametrize("source", ["p", "u", "p0"])
def test_one_point_sides(shape, source):
    check(make_case(shape, seed=sum(shape), source=source))


@pytest.mark.parametrize("shape", [(64, 1), (1, 30), (48, 40, 1), (1, 20, 18)])
def test_elastic_one_point_sides(shape):
    import kwave_b200 as kb
    import kwave_ref as K
    rng = np.random.Generator(np.random.PCG64(6))
    cp, cs, rho = (lo + (hi - lo) * rng.random(shape) for lo, hi in ((2600, 3200), (1100, 1600), (1600, 2100)))
    p0 = 1e5 * rng.random(shape)

    def run(mod):
        g = mod.KWaveGrid(*[v for n in shape for v in (n, 2e-4)])
        g.dt, g.Nt = 0.3 * 2e-4 / 3200.0, 40
        g.t_array = np.arange(40) * g.dt
        fn = mod.pstd_elastic_2d if len(shape) == 2 else mod.pstd_elastic_3d
        return fn(g, mod.ElasticMedium(sound_speed_compression=cp, sound_speed_shear=cs, density=rho),
                  mod.ElasticSource(p0=p0), mod.KWaveSensor(mask=np.ones(shape, dtype=bool), record=["p_final", "u_max"]),
                  pml_size=0)

    assert_parity(run(kb), run(K), TOL_L2, TOL_MAX)


@pytest.mark.parametrize("other", ["read", "create"])
def test_reading_a_busy_simulation_holds_up_no_other_thread(other):
    """pressure() of a simulation with a long queue of steps (40000 at 512^2, half a second) waits for them;
    a second thread that reads an idle simulation of the same context, or creates one whose fields go
    through the pinned buffer (8 MiB), is done before the first has its field."""
    import kwave_b200 as kb

    def sim(n):
        rng = np.random.default_rng(n)
        g = kb.KWaveGrid(n, 1e-4, n, 1e-4)
        g.dt, g.Nt = 2e-8, 10 ** 6
        return kb.Simulation(g, kb.KWaveMedium(sound_speed=1500.0 + 10.0 * rng.random((n, n)), density=1000.0),
                             kb.KWaveSource(p0=1e5 * rng.random((n, n))), kb.KWaveSensor())

    busy, idle = sim(512), sim(512)
    sim(1024).close()  # its schedule is measured now
    for s in (busy, idle):
        s.advance(64)
        s.sync()
    alone = idle.pressure()
    order, field, queued = [], {}, threading.Event()

    def long_read():
        busy.advance(40000)
        queued.set()
        field["busy"] = busy.pressure()
        order.append("busy")

    th = threading.Thread(target=long_read)
    th.start()
    queued.wait()
    if other == "read":
        field["idle"] = idle.pressure()
    else:
        sim(1024).close()
    order.append("other")
    th.join()
    assert order == ["other", "busy"]
    if other == "read":
        assert np.array_equal(field["idle"], alone)
    assert np.array_equal(busy.pressure(), field["busy"]) and np.isfinite(field["busy"]).all()
    busy.close()
    idle.close()


def elastic_step_us(shape, steps=64, repeats=6):
    """Device time of one step of a heterogeneous elastic simulation, the best of a few runs."""
    import kwave_b200 as kb
    rng = np.random.default_rng(2)
    g = kb.KWaveGrid(*[v for n in shape for v in (n, 2e-4)])
    g.dt, g.Nt = 0.3 * 2e-4 / 3200.0, 10 ** 6
    sim = kb.Simulation(g, kb.ElasticMedium(sound_speed_compression=2600.0 + 600.0 * rng.random(shape),
                                            sound_speed_shear=1100.0 + 500.0 * rng.random(shape),
                                            density=1600.0 + 500.0 * rng.random(shape)),
                        kb.ElasticSource(p0=1e5 * rng.random(shape)), kb.KWaveSensor(), pml_size=10)
    sim.advance(steps)
    sim.sync()
    us = min(sim.advance_timed(steps) for _ in range(repeats)) / steps * 1e3
    sim.close()
    return us


def test_narrow_elastic_tiles_are_the_faster_ones_where_the_size_rule_takes_them(monkeypatch):
    """Without a measured schedule (a batch) a 1024^2 elastic grid takes the narrow tiles: 66 us a step, the
    full-width ones 77.  With too few registers to load its running sums ahead a narrow tile took 81."""
    monkeypatch.setenv("KWB_TUNE", "0")
    us = {}
    for tile in ("big", "small"):
        monkeypatch.setenv("KWB_TILE", tile)
        us[tile] = elastic_step_us((1024, 1024))
    assert us["small"] < 0.97 * us["big"], us


# long in-place lines leave a slot free after every 16 positions (last radix 16): 1024 points in 1-D, 2048
# and 1536 along either axis, one line pair a tile and several, the transforms of a long prime side
# (1021: length 2048 or more) and the same lengths without gaps in between
@pytest.mark.parametrize("shape", [(1024,), (2048,), (4096,), (2048, 6), (6, 2048), (1536, 40), (40, 1536), (1021, 9),
                                   (9, 1021), (2048, 4, 3), (3, 4, 2048), (2000, 9)])
@pytest.mark.parametrize("stokes", [False, True])
def test_long_lines_with_gaps(shape, stokes):
    check(make_case(shape, seed=sum(shape), stokes=stokes, source="p0", steps=30))


@pytest.mark.parametrize("shape", [(2048, 12), (12, 2048), (4000, 6), (6, 4096), (1021, 10)])
def test_elastic_long_lines(shape):
    import kwave_b200 as kb
    import kwave_ref as K
    rng = np.random.Generator(np.random.PCG64(8))
    cp, cs, rho = (lo + (hi - lo) * rng.random(shape) for lo, hi in ((2600, 3200), (1100, 1600), (1600, 2100)))
    p0 = 1e5 * rng.random(shape)

    def run(mod):
        g = mod.KWaveGrid(*[v for n in shape for v in (n, 2e-4)])
        g.dt, g.Nt = 0.3 * 2e-4 / 3200.0, 25
        g.t_array = np.arange(25) * g.dt
        return mod.pstd_elastic_2d(g, mod.ElasticMedium(sound_speed_compression=cp, sound_speed_shear=cs, density=rho),
                                   mod.ElasticSource(p0=p0),
                                   mod.KWaveSensor(mask=np.ones(shape, dtype=bool), record=["p_final", "u_max"]), pml_size=2)

    assert_parity(run(kb), run(K), TOL_L2, TOL_MAX)


def test_a_line_with_many_sensor_groups_has_a_measured_schedule(monkeypatch, tmp_path):
    """More than eight recorded groups go pass by pass, with the schedule of their shape measured; eight run
    in one launch.  Every group records the same."""
    import kwave_b200 as kb
    for k in ("KWB_TUNE", "KWB_TUNE_PICK", "KWB_TUNE_ORDER", "KWB_TILE"):
        monkeypatch.delenv(k, raising=False)
    n = 1100
    case = make_case((n,), source="p0", steps=40)
    g, m, s, _, kw = case.to_api()
    mask = np.zeros(n, dtype=bool)
    mask[3::7] = True
    sensor = kb.KWaveSensor(mask=mask, record=["p_max", "p_final"])
    outs = []
    for extra, launches, src in ((7, 1, "heuristic"), (8, 12, "tuned")):
        sim = kb.Simulation(g, m, s, sensor, extra_sensors=[sensor] * extra, **kw)
        assert sim.info()["launches_per_step"] == launches
        assert sim.schedule().startswith(src) or sim.schedule().startswith("cache") and src == "tuned", sim.schedule()
        sim.advance(sim.Nt)
        outs.append(sim.outputs())
        assert len(outs[-1].extra) == extra
        for group in outs[-1].extra:
            assert all(np.array_equal(group[f], outs[-1][f]) for f in ("p_max", "p_final"))
        sim.close()
    assert_parity(outs[1], outs[0], TOL_L2, TOL_MAX)


@pytest.mark.parametrize("shape,fill,most", [((270, 256), "1", 1.2), ((112, 112), "0", 1.45)])
def test_the_size_rule_of_a_small_grid_is_near_its_measured_schedule(shape, fill, most, monkeypatch):
    """270 x 256 without a measured schedule: 46 us a step against 45 with one.  With a thread per first-stage
    butterfly alone its strided passes had 10 elements a thread in rounds of memory latency: 64.  112^2 in
    full-width tiles, as in a batch (KWB_GRID_FILL=0), against the measured narrow ones: 64 and 49, once 82."""
    import kwave_b200 as kb
    for k in ("KWB_TUNE_PICK", "KWB_TUNE_ORDER", "KWB_TILE"):
        monkeypatch.delenv(k, raising=False)
    us = {}
    for tune in ("0", "1"):
        monkeypatch.setenv("KWB_TUNE", tune)
        monkeypatch.setenv("KWB_GRID_FILL", fill if tune == "0" else "1")
        g, m, s, sen, kw = make_case(shape, source="p0", record=("p_max",), steps=2000).to_api()
        sim = kb.Simulation(g, m, s, kb.KWaveSensor(), **kw)
        sim.advance(64)
        us[tune] = min(sim.advance_timed(64) for _ in range(6)) / 64 * 1e3
        sim.close()
    assert us["0"] < most * us["1"], us


def test_the_first_simulation_of_a_shape_waits_for_few_steps(monkeypatch):
    """What measuring the schedule of a shape costs, in time steps of it: 24 candidates of 11 steps each at
    100 x 98 x 96 elastic, and the capture of their graphs.  With 33 steps a candidate it was 1000.  (A shape
    like it goes first, so that every kernel is loaded.)"""
    import time
    import kwave_b200 as kb
    for k in ("KWB_TUNE", "KWB_TUNE_PICK", "KWB_TUNE_ORDER", "KWB_TILE", "KWB_GRID_FILL"):
        monkeypatch.delenv(k, raising=False)

    def create(shape):
        rng = np.random.default_rng(4)
        g = kb.KWaveGrid(*[v for n in shape for v in (n, 2e-4)])
        g.dt, g.Nt = 0.3 * 2e-4 / 3200.0, 10 ** 6
        med = kb.ElasticMedium(sound_speed_compression=2600.0 + 600.0 * rng.random(shape),
                               sound_speed_shear=1100.0 + 500.0 * rng.random(shape), density=1600.0 + 500.0 * rng.random(shape))
        t = time.perf_counter()
        sim = kb.Simulation(g, med, kb.ElasticSource(), kb.KWaveSensor(), pml_size=10)
        return time.perf_counter() - t, sim

    create((98, 96, 100))[1].close()
    took = []
    for _ in range(3):
        t, sim = create((100, 98, 96))
        took.append(t)
        if len(took) < 3:
            sim.close()
    assert sim.schedule().startswith("cache")
    sim.advance(32)
    step = min(sim.advance_timed(32) for _ in range(4)) / 32 * 1e-3
    sim.close()
    assert took[0] - min(took[1:]) < 600 * step, (took, step)


def test_tables_of_a_long_prime_side_do_not_dominate_its_set_up():
    """Creating a 1-D simulation of 2039 points (a prime: three tables of 4096-point transforms) against one
    of 2048.  With the tables summed term by term: 10 ms against 0.8."""
    import time
    import kwave_b200 as kb
    ms = {}
    for n in (2039, 2048):
        g, m, s, _, kw = make_case((n,), source="p0", steps=20).to_api()
        ms[n] = 1e9
        for _ in range(6):
            t = time.perf_counter()
            sim = kb.Simulation(g, m, s, kb.KWaveSensor(), **kw)
            ms[n] = min(ms[n], 1e3 * (time.perf_counter() - t))
            sim.close()
    assert ms[2039] < 4 * ms[2048], ms


# the dispersion term at half and at four times the equation of state's own (its multiplier grows as
# k^(y-1) / dt, and with tan(pi y/2) near y = 1), on grids fine enough and with steps short enough for the
# scheme itself to be stable; also a step at a time, nonlinear, and with a Bluestein side.  Tolerance: the error
# of the FP32 oracle, whose dispersion term transforms the change of the density, half as much again.
@pytest.mark.parametrize("shape", [(512,), (60, 45), (64, 96), (34, 40), (20, 22, 18)])
@pytest.mark.parametrize("dx,cfl,y,nonlinear", [(1e-4, 0.3, 1.02, False), (1e-5, 0.1, 1.5, False), (1e-5, 0.1, 1.5, True)])
def test_strong_dispersion(shape, dx, cfl, y, nonlinear):
    if len(shape) == 3 and y == 1.02:
        dx, cfl = 2e-4, 0.2
    l2 = {}
    for seed in (11, 12, 13):
        case = make_case(shape, seed=seed, stokes=True, source="p0", steps=120, record=("p_final",), nonlinear=nonlinear)
        case.medium["alpha_power"] = y
        case.d, case.dt = (dx,) * len(shape), cfl * dx / 1500.0
        ref = run_oracle(case)
        for name, out in (("gpu", run_gpu(case)), ("fp32", run_oracle(case, dtype=np.float32))):
            l2[name] = l2.get(name, 0.0) + errors(out["p_final"], ref["p_final"])[0]
    assert l2["gpu"] < 1.5 * l2["fp32"], l2


@pytest.mark.parametrize("n", [96, 1024, 2401, 34])
def test_strong_dispersion_of_a_line_in_pieces(n):
    """In one launch and pass by pass (profile), in turn; 34 points go pass by pass throughout."""
    import kwave_b200 as kb
    case = make_case((n,), source="p0", stokes=True, record=("p",), steps=90)
    case.d, case.dt = (1e-5,), 1e-6 / 1500.0
    g, m, s, sen, kw = case.to_api()
    sim = kb.Simulation(g, m, s, sen, **kw)
    assert sim.info()["launches_per_step"] == (5 if n == 34 else 1)
    sim.advance(1)
    sim.profile(5)
    sim.advance(33)
    assert_parity(sim.finish(), run_oracle(case), TOL_L2, TOL_MAX)
    sim.close()


# the register passes hold up to 96 source entries of a tile in shared memory, up to three a thread in the
# narrowest, and read more in place: counts at that edge, all of them on the lines of one tile, which are at
# least 8 consecutive rows (x) of 64 points or 4 columns (y) of 128
@pytest.mark.parametrize("points", [32, 33, 95, 96, 97, 200])
@pytest.mark.parametrize("tile", ["big", "mid", "small"])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("source,mode", [("p", 0), ("u", 1)])
def test_source_entries_at_the_edge_of_a_tile(points, tile, axis, source, mode, monkeypatch):
    monkeypatch.setenv("KWB_TILE", tile)
    shape = (64, 128)
    case = make_case(shape, seed=points, source=source, points=1, mode=mode, steps=20)
    rng = np.random.Generator(np.random.PCG64(points))
    rows = np.zeros(shape, dtype=bool)  # the lines of a tile: rows y < 8 of the x pass, columns x < 4 of the y pass
    rows[(slice(None), slice(0, 8)) if axis == 0 else (slice(0, 4), slice(None))] = True
    mask = np.zeros(shape, dtype=bool)
    mask.reshape(-1)[rng.choice(np.flatnonzero(rows), points, replace=False)] = True
    sig = 1e5 * rng.standard_normal((points, 12))
    case.source = dict(p_mask=mask, p=sig, p_mode=mode) if source == "p" else dict(
        u_mask=mask, u_mode=mode, ux=1e-6 * sig, uy=-1e-6 * sig)
    check(case)
