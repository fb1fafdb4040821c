"""Edges of the accepted range: grids with one-point sides.

Tolerance as in test_gpu_any_length.py: about ten transforms a step, each adding some 2e-7 of relative
rounding error, below 3e-5 over 60 steps.
"""
import numpy as np
import pytest

from _util import assert_parity
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
