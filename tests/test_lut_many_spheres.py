"""The sorted mixed LUT kernel (more than 8 spheres) at the edges of its ranges, and the plain kernel beside it,
against the oracle with the parity suite's mixed tolerances (1e-5 on the detector images,
1e-4 on the near field); staged against unstaged, and tables in pieces against one piece, bit for bit."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_IMG_INTENSITY, BS_PREC_MIXED, Context, abi, scenes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def spheres(ns, fov, first=()):
    rest = [(fov * (0.04 + 0.92 * (i + 0.5) / ns - 0.5), fov * (0.37 * i % 1 - 0.5), 0.1 * (i % 5), 0.02 * fov * (1 + i % 3),
             1.3 + 0.01 * (i % 20), 0.01) for i in range(ns - len(first))]
    return list(first) + rest


def run(p, s, w, staging=0, budget=0):
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.set_lut_staging(staging)
        if budget:
            ctx.set_lut_budget(budget)
        ctx.simulate(BS_PREC_MIXED)
        return ctx.field(), ctx.image(BS_IMG_INTENSITY, f64=True), ctx.stats()


def check(p, s, w):
    U, _, D, _ = oracle_lib.simulate(p, *abi.sphere_array(s), w)
    a, b = run(p, s, w), run(p, s, w, staging=2)
    assert rel(a[0], U) <= 1e-4 and rel(a[1], D) <= 1e-5, (rel(a[0], U), rel(a[1], D))
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    return a


# directions: the counts around the plain kernel's largest, a part group, exactly one and one more than one sort
# block of 1024, two part blocks; spheres: the plain kernel's largest count and one more
@pytest.mark.parametrize("nk", [1, 31, 32, 33, 63, 64, 65, 95, 1024, 1025, 1500])
@pytest.mark.parametrize("ns", [8, 9])
def test_direction_counts(ns, nk):
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(24, 0), resolution=12, padding=1,
                        us_lut_r=120, us_lut_theta=300)
    check(p, spheres(ns, 24), scenes.mc_waves(nk, 0, 0.5, seed=21))


# rows of a part tile, polynomial rows at fine pitch and arc cosines at coarse pitch, directions through the poles,
# more columns than a window for every group, an odd column count, a plane of another direction
@pytest.mark.parametrize("kw", [
    dict(xy=(6, 0), resolution=11, us_lut_theta=1024),
    dict(xy=(150, 0), resolution=13, us_lut_theta=1024),
    dict(xy=(12, 3.0), resolution=13, condenser=(0, 1.0), us_lut_theta=400),
    dict(xy=(24, 0), resolution=16, us_lut_theta=3001),
    dict(plane=((-8, 0.5, -8), (8, 0.5, 8), (0, -1, 0)), resolution=13, us_lut_theta=200),
])
def test_geometries(kw):
    kw = dict(dict(condenser=(0, 0.5)), **kw)
    p = abi.make_params(lam=2.5, objective=(0, 0.5), padding=1, us_lut_r=150, supersample=1, **kw)
    first = [(0.0, 0.0, 0.0, 1.5, 1.45, 0.03), (2.6, -2.2, 0.4, 0.8, 1.3, 0.0)]
    check(p, spheres(9, 12, first), scenes.mc_waves(200, *kw["condenser"], seed=22))


def test_directions_that_are_not_unit_vectors():
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(24, 0), resolution=12, padding=1,
                        us_lut_r=120, us_lut_theta=300)
    w = scenes.mc_waves(100, 0, 0.5, seed=23) * np.linspace(0.9, 1.3, 100)[:, None]
    assert check(p, spheres(9, 24), w)[2].lut_chunks_staged == 0


# columns as in the forward-direction test: the row of pixels through a sphere's centre has cosine 1
@pytest.mark.parametrize("theta", [256, 400, 700, 1024])
def test_pixels_straight_behind_a_sphere(theta):
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), plane=((-4, 0, -4), (4, 0, 4), (0, 1, 0)),
                        resolution=12, padding=1, us_lut_r=400, us_lut_theta=theta)
    s = spheres(9, 4, [(0.0, 0.0, 0.0, 1.0, 1.4, 0.01)])
    w = scenes.mc_waves(200, 0, 0.5, seed=41)
    w[100] = (0.0, 0.0, 1.0)
    U = oracle_lib.simulate(p, *abi.sphere_array(s), w)[0]
    err = np.abs(check(p, s, w)[0] - U) / np.abs(U).max()
    assert err.max() <= 1e-4, (err.max(), np.argwhere(err > 1e-4)[:8].tolist())


# shares of one sphere each (16), one share of two (17), of two and three (37); tables in one piece and in pieces of
# about two and a half spheres, whose edges lie inside shares
@pytest.mark.parametrize("ns", [16, 17, 37])
def test_shares_of_several_spheres(ns):
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(40, 0), resolution=19, padding=1,
                        us_lut_r=120, us_lut_theta=400)
    s, w = spheres(ns, 40), scenes.mc_waves(130, 0, 0.5, seed=31)
    whole = check(p, s, w)
    pieces = run(p, s, w, budget=int(2.5 * 140 * 402 * 8))
    assert np.array_equal(whole[0], pieces[0]) and np.array_equal(whole[1], pieces[1])
