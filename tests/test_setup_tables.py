"""The setup kernels (Mie coefficients, coefficient rows, harmonics' tables) at the edges of their ranges,
against the oracle: double precision to the parity suite's 1e-10."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_IMG_INTENSITY, BS_PREC_FP64, Context, abi, scenes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def check(s, nk, **kw):
    kw = dict(dict(lam=1.0, condenser=(0, 0.4), objective=(0, 0.4), resolution=7, padding=1, supersample=1,
                   us_lut_r=45, us_lut_theta=70), **kw)
    p = abi.make_params(**kw)
    w = scenes.mc_waves(nk, 0, 0.4, seed=61)
    U, _, D, _ = oracle_lib.simulate(p, *abi.sphere_array(s), w)
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.simulate(BS_PREC_FP64)
        f, d = ctx.field(), ctx.image(BS_IMG_INTENSITY, f64=True)
    assert rel(f, U) <= 1e-10 and rel(d, D) <= 1e-10, (rel(f, U), rel(d, D))


# a sphere of few orders; one of about 110 (values of a block above 48 KB of shared memory); one that absorbs so
# strongly that the start order of the recurrence is the long one; spheres of all three kinds, whose rows share
# blocks and whose block edges fall inside a sphere's rows
SMALL, LARGE, DARK = (2.0, 1.0, 0.0, 0.02, 1.5, 0.0), (-3.0, 2.0, 0.5, 12.0, 1.3, 0.001), (1.0, -2.0, 0.3, 5.0, 1.4, 1.1)


@pytest.mark.parametrize("s,fov,z", [([SMALL], 6, 0.0), ([LARGE], 40, 0.5), ([DARK], 16, 0.0),
                                     ([SMALL, (8.0, 9.0, 0.0, 5.0, 1.4, 1.1), (-9.0, -3.0, 0.2, 3.0, 1.5, 0.02)], 30, 0.1)])
def test_rows(s, fov, z):
    check(s, 9, xy=(fov, z))


# harmonics of fewer orders than a warp and of more than one and than three, directions below, at and above a
# warp and not a multiple of 16, planes through the centre and beside it
@pytest.mark.parametrize("s,fov,z,nk", [([SMALL], 6, 0.0, 1), ([(0.5, 0.3, 0.0, 2.5, 1.4, 0.01)], 12, 0.0, 32),
                                        ([(0.5, 0.3, 0.0, 3.6, 1.4, 0.01)], 16, 0.7, 33), ([LARGE], 40, 0.5, 50),
                                        ([LARGE], 40, 1.5, 5)])
def test_harmonics(s, fov, z, nk):
    check(s, nk, xy=(fov, z), lut_us=False, lut_uf=False)


# scenes of eight spheres whose inner rows, those scaled by j_1, share blocks with other spheres' outer rows
@pytest.mark.parametrize("seed", [16, 21, 23])
def test_rows_of_many_spheres(seed):
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(24, 0), resolution=96, padding=1,
                        supersample=1)
    s = scenes.random_spheres(8, 24.0, 0.8, 2.5, seed=seed * 1009 + 2, z_slab=0.0)
    w = scenes.mc_waves(6, 0, 0.5, seed=seed)
    U = oracle_lib.simulate(p, *abi.sphere_array(s), w)[0]
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.simulate(BS_PREC_FP64)
        assert rel(ctx.field(), U) <= 1e-10
