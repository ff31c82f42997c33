"""The folded double-precision forward transforms against the oracle, to the parity suite's 1e-10, and the short
single-precision ones to its 1e-5."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_IMG_INCIDENT, BS_IMG_INTENSITY, BS_PREC_FP64, BS_PREC_MIXED, Context, abi, scenes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


# near-field sizes R with and without a sample R / 2 (alone in its pair), of one tile of 32 rows and folded samples
# and a few more; passbands of the bin 0 alone, of fewer and more bins than a tile, and of every bin (pixels of 2 um
# at 1 um: above the Nyquist frequency); an annulus
@pytest.mark.parametrize("res,ss,fov,na", [(3, 1, 2.0, (0, 0.2)), (8, 1, 16.0, (0, 0.5)), (11, 1, 22.0, (0, 0.8)),
                                           (11, 2, 12.0, (0, 0.5)), (21, 1, 10.0, (0.2, 0.6)), (16, 3, 30.0, (0, 0.7)),
                                           (43, 3, 40.0, (0, 0.9))])
def test_passbands(res, ss, fov, na):
    p = abi.make_params(lam=1.0, condenser=(0, 0.4), objective=na, xy=(fov, 0.5), resolution=res, padding=1,
                        supersample=ss, us_lut_r=60, us_lut_theta=100)
    s = [(0.1 * fov, -0.05 * fov, 0.0, 0.7, 1.4, 0.02)]
    w = scenes.mc_waves(12, 0, 0.4, seed=51)
    _, _, D, Di = oracle_lib.simulate(p, *abi.sphere_array(s), w)
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.simulate(BS_PREC_FP64)
        d, di = ctx.image(BS_IMG_INTENSITY, f64=True), ctx.image(BS_IMG_INCIDENT, f64=True)
    assert rel(d, D) <= 1e-10 and rel(di, Di) <= 1e-10, (rel(d, D), rel(di, Di))


# single-precision transforms of at most 64 rows, columns and products (near fields of 63 pixels), and of one more
@pytest.mark.parametrize("res", [1, 21, 22])
def test_short_float_transforms(res):
    p = abi.make_params(lam=1.0, condenser=(0, 0.4), objective=(0, 0.7), xy=(0.5 * res, 0.5), resolution=res, padding=1,
                        supersample=1, us_lut_r=60, us_lut_theta=200)
    s = [(0.05 * res, -0.02 * res, 0.0, 0.7, 1.4, 0.02)]
    w = scenes.mc_waves(40, 0, 0.4, seed=52)
    _, _, D, Di = oracle_lib.simulate(p, *abi.sphere_array(s), w)
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.simulate(BS_PREC_MIXED)
        d, di = ctx.image(BS_IMG_INTENSITY, f64=True), ctx.image(BS_IMG_INCIDENT, f64=True)
    assert rel(d, D) <= 1e-5 and rel(di, Di) <= 1e-5, (rel(d, D), rel(di, Di))
