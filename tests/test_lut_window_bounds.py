"""Window bounds of the mixed LUT kernels where single precision is short: every lookup has to lie in its window, so the
staged kernel gives the bits of the unstaged one and the oracle's field (1e-4 of the largest, pixel by
pixel)."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_PREC_MIXED, Context, abi, scenes

pytestmark = pytest.mark.gpu


def check(p, s, w):
    U = oracle_lib.simulate(p, *abi.sphere_array(s), w)[0]
    got = []
    for staging in (0, 2):
        with Context(p) as ctx:
            ctx.set_spheres(s)
            ctx.set_waves(w)
            ctx.set_lut_staging(staging)
            ctx.simulate(BS_PREC_MIXED)
            got.append((ctx.field(), ctx.stats().lut_chunks_staged))
    err = np.abs(got[0][0] - U) / np.abs(U).max()
    assert err.max() <= 1e-4, (err.max(), np.argwhere(err > 1e-4)[:8].tolist())
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1] > 0


# a slice and its spheres 1e6 to 1e8 um from the origin: positions in single precision are 0.06 to 8 um apart
@pytest.mark.parametrize("far", [0.0, 1e6, 1e7, 1e8])
@pytest.mark.parametrize("ns", [8, 9])
def test_slices_far_from_the_origin(far, ns):
    o = np.array([far, -0.6 * far, 0.3 * far])
    h = 0.8
    p = abi.make_params(lam=2.5, condenser=(0, 0.5), objective=(0, 0.5), resolution=32, padding=1, supersample=1,
                        us_lut_r=120, us_lut_theta=1024, plane=(tuple(o - (h, h, 0)), tuple(o + (h, h, 0)), (0.0, 0.0, 1.0)))
    p.focus[:] = list(o)
    s = [(o[0] + 1.1 * (i % 3) - 1.2, o[1] + 1.3 * (i // 3) - 1.1, o[2] - 15.0 + 0.2 * (i % 2), 0.3 + 0.02 * i, 1.35, 0.01)
         for i in range(ns)]
    check(p, s, scenes.mc_waves(400, 0, 0.5, seed=7))


# directions up to 1e-6 longer or shorter than 1, as decimal files hold them, along the lines from spheres to pixels,
# in tables of 0.0001 rad a column: the angle of a direction of length 1.000001 is off by up to 13 columns
@pytest.mark.parametrize("length", [1.0, 1 + 9.9e-7, 1 - 9.9e-7])
@pytest.mark.parametrize("ns", [8, 9])
def test_directions_of_almost_unit_length(length, ns):
    p = abi.make_params(lam=2.5, condenser=(0, 0.004), objective=(0, 0.5), resolution=32, padding=1, supersample=1,
                        us_lut_r=20, us_lut_theta=30000, xy=(0.08, 15.0))
    s = [(0.01 * (i % 3) - 0.01, 0.01 * (i // 3) - 0.01, 0.5 * i - 2.0, 0.2 + 0.01 * i, 1.35, 0.01) for i in range(ns)]
    check(p, s, length * scenes.mc_waves(256, 0, 0.004, seed=8))
