"""Directions that pass exactly through a sphere's centre and pixels (cosine 1, table column 0), against the
oracle: every pixel's near field to the mixed tolerance 1e-4 of the largest."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_PREC_MIXED, Context, abi, scenes

pytestmark = pytest.mark.gpu


# column counts whose half turn in columns, rounded, is below pi / 2 times the rounded column scale (256, 700, 1024)
# and above it (400); one thread per pixel (20 directions) and the sorted kernel
@pytest.mark.parametrize("theta", [256, 400, 700, 1024])
@pytest.mark.parametrize("nk", [20, 33, 200])
@pytest.mark.parametrize("staging", [0, 2])
def test_pixels_straight_behind_the_sphere(theta, nk, staging):
    # rows of pixels along z, the axis of the directions: the row through the sphere has cosine 1
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), plane=((-4, 0, -4), (4, 0, 4), (0, 1, 0)),
                        resolution=12, padding=1, us_lut_r=400, us_lut_theta=theta)
    s = [(0.0, 0.0, 0.0, 2.0, 1.4, 0.01)]
    w = scenes.mc_waves(nk, 0, 0.5, seed=41)
    w[nk // 2] = (0.0, 0.0, 1.0)
    U = oracle_lib.simulate(p, *abi.sphere_array(s), w)[0]
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.set_lut_staging(staging)
        ctx.simulate(BS_PREC_MIXED)
        f = ctx.field()
    err = np.abs(f - U) / np.abs(U).max()
    assert err.max() <= 1e-4, (err.max(), np.argwhere(err > 1e-4)[:8].tolist())
