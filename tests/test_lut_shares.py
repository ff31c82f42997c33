"""The mixed LUT kernel's shares of the spheres on grids of few tiles and its window shapes, against
the oracle with the parity suite's mixed tolerances (1e-5 on the detector images, 1e-4 on the near
field), staged against unstaged bit for bit."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_IMG_INTENSITY, BS_PREC_MIXED, Context, abi, scenes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


# spheres: one (no shares), fewer than the most shares (8), one more, shares of unequal size; tables in one piece
# and, with room for about two spheres, in pieces whose edges are not those of the shares.  Pitches from windows of
# 16 pixels x 64 columns (10 um) to 8 x 128 and 4 x 256 (40 um) and cells read from the table (100 um).
@pytest.mark.parametrize("ns,fov,pieces", [(1, 40, False), (2, 10, True), (3, 40, True), (8, 100, False),
                                           (9, 40, False), (11, 20, True)])
def test_shares(ns, fov, pieces):
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(fov, 0), resolution=19, padding=1,
                        us_lut_r=120, us_lut_theta=1024)
    s = [(fov * (0.04 + 0.083 * i - 0.5), fov * (0.37 * i % 1 - 0.5), 0.1 * i, 0.6 + 0.13 * i, 1.3 + 0.01 * i, 0.01)
         for i in range(ns)]
    w = scenes.mc_waves(330, 0, 0.5, seed=31)
    U, _, D, _ = oracle_lib.simulate(p, *abi.sphere_array(s), w)
    got = []
    for staging in (0, 2):
        with Context(p) as ctx:
            ctx.set_spheres(s)
            ctx.set_waves(w)
            ctx.set_lut_staging(staging)
            if pieces:
                ctx.set_lut_budget(int(2.5 * 120 * 1024 * 8))
            ctx.simulate(BS_PREC_MIXED)
            got.append((ctx.field(), ctx.image(BS_IMG_INTENSITY, f64=True)))
    assert rel(got[0][0], U) <= 1e-4 and rel(got[0][1], D) <= 1e-5, (rel(got[0][0], U), rel(got[0][1], D))
    assert np.array_equal(got[0][0], got[1][0])


def test_ranges():
    """A grid too large for shares with tables of twice 256 MB: two launches, the bits of a table at a time."""
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(60, 0), resolution=529, padding=1,
                        supersample=1, us_lut_r=4096, us_lut_theta=1024)
    s = [(14 * (i % 4) - 21.0, 14 * (i // 4) - 22.0, 0.0, 1.0, 1.3 + 0.01 * i, 0.01) for i in range(16)]
    w = scenes.mc_waves(40, 0, 0.5, seed=32)
    got = []
    for budget in (0, 40 << 20):
        with Context(p) as ctx:
            ctx.set_spheres(s)
            ctx.set_waves(w)
            if budget:
                ctx.set_lut_budget(budget)
            ctx.simulate(BS_PREC_MIXED)
            got.append((ctx.field(), ctx.stats().kernel_launches))
    assert got[0][1] < got[1][1]
    assert np.array_equal(got[0][0], got[1][0])
