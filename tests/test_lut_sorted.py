"""The mixed LUT kernel at the edges of its ranges, against the oracle with the parity suite's
mixed tolerances (1e-5 on the detector images, 1e-4 on the near field), and staged against
unstaged bit for bit."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_IMG_INTENSITY, BS_PREC_MIXED, Context, abi, scenes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def run(p, s, w, staging=0):
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.set_lut_staging(staging)
        ctx.simulate(BS_PREC_MIXED)
        return ctx.field(), ctx.image(BS_IMG_INTENSITY, f64=True), ctx.stats()


# directions: the largest count of one thread per pixel (32), the smallest of the sorted kernel (33), a part
# group, exactly one and one more than one sort block of 1024, two part blocks
@pytest.mark.parametrize("nk", [32, 33, 95, 1024, 1025, 1500])
def test_direction_counts(nk):
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(24, 0), resolution=12, padding=1,
                        us_lut_r=120, us_lut_theta=300)
    s = [(1.0, -2.0, 0.0, 2.0, 1.4, 0.04), (-6.0, 5.0, 1.0, 1.2, 1.5, 0.01)]
    w = scenes.mc_waves(nk, 0, 0.5, seed=21)
    U, _, D, _ = oracle_lib.simulate(p, *abi.sphere_array(s), w)
    a, b = run(p, s, w), run(p, s, w, staging=2)
    assert rel(a[0], U) <= 1e-4 and rel(a[1], D) <= 1e-5
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


# geometries: rows of a part tile (R = 33, 39), polynomial rows at fine pitch (fov 6) and arc cosines at coarse
# pitch (fov 150), directions through the poles (a plane above the spheres, a condenser up to NA 1), a sphere
# centred on a pixel, a table with more columns than a window for every group
@pytest.mark.parametrize("kw", [
    dict(xy=(6, 0), resolution=11, us_lut_theta=1024),
    dict(xy=(150, 0), resolution=13, us_lut_theta=1024),
    dict(xy=(12, 3.0), resolution=13, condenser=(0, 1.0), us_lut_theta=400),
    dict(xy=(24, 0), resolution=16, us_lut_theta=3000),
    dict(plane=((-8, 0.5, -8), (8, 0.5, 8), (0, -1, 0)), resolution=13, us_lut_theta=200),
])
def test_geometries(kw):
    kw = dict(dict(condenser=(0, 0.5)), **kw)
    p = abi.make_params(lam=2.5, objective=(0, 0.5), padding=1, us_lut_r=150, supersample=1, **kw)
    s = [(0.0, 0.0, 0.0, 1.5, 1.45, 0.03), (2.6, -2.2, 0.4, 0.8, 1.3, 0.0)]
    w = scenes.mc_waves(200, *kw["condenser"], seed=22)
    U, _, D, _ = oracle_lib.simulate(p, *abi.sphere_array(s), w)
    a, b = run(p, s, w), run(p, s, w, staging=2)
    assert rel(a[0], U) <= 1e-4 and rel(a[1], D) <= 1e-5, (rel(a[0], U), rel(a[1], D))
    assert np.array_equal(a[0], b[0])


def test_directions_that_are_not_unit_vectors():
    """Scaled directions: the angle clamps at 0 and pi, no angle bound holds, nothing is staged."""
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(24, 0), resolution=12, padding=1,
                        us_lut_r=120, us_lut_theta=300)
    s = [(1.0, -2.0, 0.0, 2.0, 1.4, 0.04)]
    w = scenes.mc_waves(100, 0, 0.5, seed=23) * np.linspace(0.9, 1.3, 100)[:, None]
    U, _, D, _ = oracle_lib.simulate(p, *abi.sphere_array(s), w)
    f, d, st = run(p, s, w)
    assert st.lut_chunks_staged == 0
    assert rel(f, U) <= 1e-4 and rel(d, D) <= 1e-5
