"""The mixed path's table build at the edges of its tiles: rows around 32, angles around 128, orders around
16, a Uip of one row, against the oracle's double-precision tables.  A float entry is within half an ulp
of its value: 6e-8 relative to the largest entry bounds every one, 2e-7 leaves room for the build."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_PREC_MIXED, Context, abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,theta,a", [(31, 127, 0.4), (32, 128, 1.3), (33, 129, 2.7), (65, 257, 6.0), (2, 2, 1.0)])
def test_tables_at_tile_edges(rows, theta, a):
    p = abi.make_params(lam=2.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(30, 0), resolution=8, padding=1,
                        us_lut_r=rows, us_lut_theta=theta)
    s = [(0.5, -0.3, 0.0, a, 1.45, 0.03), (9.0, 8.0, 3.0, 0.5 * a, 1.3, 0.0)]  # the second: Uip of one row if a < 6
    lib = oracle_lib.load()
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(scenes.mc_waves(8, 0, 0.5, seed=3))
        ctx.simulate(BS_PREC_MIXED)
        for i, sp in enumerate(s):
            g = oracle_lib.sphere_geom(p, abi.Sphere(*sp))
            ref = [np.zeros(2 * g.dR * g.thetaR), np.zeros(2 * g.aR * g.thetaR)]
            lib.bso_sphere_luts(oracle_lib.C.byref(p), oracle_lib.C.byref(abi.Sphere(*sp)), oracle_lib.P(ref[0]),
                                oracle_lib.P(ref[1]))
            for which, n in ((0, g.dR), (1, g.aR)):
                r = ref[which].view(np.complex128).reshape(n, theta)
                assert np.abs(ctx.lut(i, which, n, theta) - r).max() <= 2e-7 * np.abs(r).max()
