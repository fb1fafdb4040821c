"""The passes that serve any line length, and the branches of the register passes beside them, against
the FP64 oracle at the lengths and counts where they can go wrong.

Tolerance: a step takes about ten transforms, each adding some 2e-7 of relative rounding error in
FP32 (log2 N levels of 6e-8, in quadrature); over 60 steps, with the errors of different steps added
in quadrature or, at worst, a fifth of them coherently, that is below 3e-5.
"""
import numpy as np
import pytest

from _util import assert_parity, run_gpu, run_oracle

pytestmark = pytest.mark.gpu

TOL_L2, TOL_MAX = 3e-5, 3e-4
STEPS = 60


def make_case(shape, seed=1, stokes=False, mode=1, source="p", points=5, record=("p_final", "p_rms", "u_max"), steps=STEPS,
              nonlinear=False):
    from kwave_b200.workloads import Case
    rng = np.random.Generator(np.random.PCG64(seed))
    D = len(shape)
    med = dict(sound_speed=1500.0, density=1000.0) if stokes else dict(
        sound_speed=1400.0 + 200.0 * rng.random(shape), density=900.0 + 200.0 * rng.random(shape))
    med.update(alpha_coeff=0.75, alpha_power=1.5, alpha_mode="stokes" if stokes else "no_dispersion")
    if nonlinear:
        med["BonA"] = 6.0
    src = {}
    mask = np.zeros(shape, dtype=bool)
    flat = rng.choice(mask.size, size=min(points, mask.size), replace=False)
    mask.reshape(-1)[flat] = True
    sig = 1e5 * rng.standard_normal((int(mask.sum()), 12))
    if source == "p":
        src = dict(p_mask=mask, p=sig, p_mode=mode)
    elif source == "u":
        src = {"u_mask": mask, "u_mode": mode, **{c: 0.1 * 1e-5 * sig for c in ("ux", "uy", "uz")[:D]}}
    else:
        p0 = rng.random(shape)
        src = dict(p0=1e5 * p0)
    sensor = dict(mask=np.ones(shape, dtype=bool), record=list(record))
    return Case("any", shape, (1e-4,) * D, 0.3 * 1e-4 / 1600.0, steps, med, src, sensor, pml_size=min(4, min(shape) // 4))


def check(case):
    assert_parity(run_gpu(case), run_oracle(case), TOL_L2, TOL_MAX)


# one stage (13, 16), two and three with every radix, four (7^4 on its own is 1-D), odd and unpaired
# columns, columns not a multiple of 4, and lengths with a prime factor above 13 as convolutions
@pytest.mark.parametrize("shape", [(16, 13), (13, 16), (9, 121), (66, 65), (126, 135), (99, 34), (17, 250), (77, 62),
                                   (101, 37), (30, 343), (22, 529), (14, 15, 13), (18, 33, 20), (37, 10, 19)])
@pytest.mark.parametrize("source", ["p", "u", "p0"])
def test_any_length(shape, source):
    check(make_case(shape, seed=sum(shape), source=source))


# dispersion on the register passes (64 x 96, 32-multiple volume), on the in-place passes, with
# Bluestein equation-of-state passes along either axis, nonlinear, and the plane pass's size
@pytest.mark.parametrize("shape", [(64, 96), (96, 64), (60, 66), (34, 64), (64, 34), (64, 64, 64), (20, 22, 18)])
@pytest.mark.parametrize("nonlinear", [False, True])
def test_dispersion_from_the_last_spectrum(shape, nonlinear):
    check(make_case(shape, seed=7, stokes=True, nonlinear=nonlinear))


# the register passes hold up to 96 source entries of a tile in shared memory and read more in place
@pytest.mark.parametrize("points", [1, 40, 95, 127, 129, 2000])
@pytest.mark.parametrize("source", ["p", "u"])
@pytest.mark.parametrize("mode", [0, 1])
def test_source_entries_of_a_tile(points, source, mode):
    check(make_case((64, 128), seed=points, source=source, points=points, mode=mode))


# 1-D runs of steps in one launch: single-stage, odd and three-stage lines, both source kinds and
# modes, dispersion, every field recorded, and runs split over several calls
@pytest.mark.parametrize("n", [13, 64, 75, 512, 2401])
@pytest.mark.parametrize("source,mode,stokes", [("p", 1, False), ("p", 0, True), ("u", 0, False), ("u", 1, True),
                                                ("p0", 1, True)])
def test_steps_of_a_line(n, source, mode, stokes):
    rec = ("p", "p_max", "p_min", "p_rms", "p_final", "ux", "u_max", "u_rms", "u_final")
    check(make_case((n,), seed=n, source=source, mode=mode, stokes=stokes, record=rec, points=3))


def test_steps_of_a_line_in_pieces_and_launched_one_by_one():
    import kwave_b200 as kb
    case = make_case((96,), source="p", stokes=True, record=("p",), points=3, steps=90)
    whole = run_gpu(case)
    g, m, s, sen, kw = case.to_api()
    sim = kb.Simulation(g, m, s, sen, **kw)
    sim.advance(1)
    sim.profile(5)  # these go pass by pass
    sim.advance(33)
    out = sim.finish()
    ref = run_oracle(case)
    assert_parity(out, ref, TOL_L2, TOL_MAX)
    assert_parity(whole, ref, TOL_L2, TOL_MAX)
    sim.close()


@pytest.mark.parametrize("shape", [(512, 512), (520, 505), (64, 64, 65)])
def test_pressure_through_pinned_chunks(shape):
    """At least 2^18 points go through the pinned buffer: the same field as the sensor's p_final."""
    import kwave_b200 as kb
    case = make_case(shape, source="p", record=("p_final",), steps=12)
    g, m, s, sen, kw = case.to_api()
    sim = kb.Simulation(g, m, s, sen, **kw)
    sim.advance(sim.Nt)
    p = sim.pressure()
    assert np.array_equal(p.ravel(order="F").astype(np.float64), sim.outputs()["p_final"])
    sim.close()


@pytest.mark.parametrize("shape", [(17, 22), (15, 46), (9, 17, 12)])
def test_elastic_any_length(shape):
    import kwave_b200 as kb
    import kwave_ref as K
    rng = np.random.Generator(np.random.PCG64(5))
    cp, cs, rho = (lo + (hi - lo) * rng.random(shape) for lo, hi in ((2600, 3200), (1100, 1600), (1600, 2100)))
    p0 = 1e5 * rng.random(shape)
    D = len(shape)

    def run(mod):
        g = mod.KWaveGrid(*[v for n in shape for v in (n, 2e-4)])
        g.dt, g.Nt = 0.3 * 2e-4 / 3200.0, 40
        g.t_array = np.arange(40) * g.dt
        fn = mod.pstd_elastic_2d if D == 2 else mod.pstd_elastic_3d
        return fn(g, mod.ElasticMedium(sound_speed_compression=cp, sound_speed_shear=cs, density=rho),
                  mod.ElasticSource(p0=p0), mod.KWaveSensor(mask=np.ones(shape, dtype=bool), record=["p_final", "u_max"]),
                  pml_size=2)

    assert_parity(run(kb), run(K), TOL_L2, TOL_MAX)
