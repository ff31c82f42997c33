"""The block-per-sphere Mie kernel over its range of k a and orders, against the oracle at the parity suite's
1e-12: the smallest spheres (orders cut off below 1e-200 for the interior argument), ka at the y_0 branch of 12,
more orders than threads of a block, and step factors beyond the shared table (|n| k a near 900)."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_PREC_FP64, Context, abi, scenes

pytestmark = pytest.mark.gpu

LAM = 2.0


@pytest.mark.parametrize("a,n_re,n_im", [(0.02, 1.4, 0.05), (3.81, 1.4, 0.0), (3.83, 1.55, 0.05), (60.0, 1.2, 0.0),
                                         (100.0, 2.8, 0.0)])
def test_coefficients(a, n_re, n_im):
    lib = oracle_lib.load()
    nl = lib.bso_calc_nl(a, LAM)
    p = abi.make_params(lam=LAM, condenser=(0, 0.5), objective=(0, 0.5), xy=(400, 0), resolution=2, padding=0,
                        supersample=1, us_lut_r=4, us_lut_theta=4)
    with Context(p) as ctx:
        ctx.set_spheres([(0, 0, 0, a, n_re, n_im)])
        ctx.set_waves(scenes.mc_waves(4, 0, 0.5, seed=1))
        ctx.simulate(BS_PREC_FP64)
        A, B = ctx.mie(0, nl)
    ref = [np.zeros(2 * nl + 2), np.zeros(2 * nl + 2)]
    lib.bso_mie(2 * float(np.float32(3.14159)) / LAM, a, n_re, n_im, nl, oracle_lib.P(ref[0]), oracle_lib.P(ref[1]))
    for got, r in ((A, ref[0]), (B, ref[1])):
        r = r.view(np.complex128)
        assert np.linalg.norm(got - r) <= 1e-12 * np.linalg.norm(r)
