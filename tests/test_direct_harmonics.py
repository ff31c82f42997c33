"""The direct method with the harmonics about the slice's normal: spheres centred in the plane (constant
harmonics) and beside it in one scene, planes along every axis and an oblique one, a slice that is a line, a
pixel at a sphere's centre; double precision against the oracle's sums over directions (1e-10)."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_PREC_FP64, Context, abi, scenes

pytestmark = pytest.mark.gpu

PLANES = {
    "xy": ((-6, -6, 0.5), (6, 6, 0.5), (0, 0, 1)),
    "xz": ((-6, 0.5, -6), (6, 0.5, 6), (0, 1, 0)),
    "yz": ((0.5, -6, -6), (0.5, 6, 6), (1, 0, 0)),
    "oblique": ((-5, -5, -2.5), (5, 5, 3.5), tuple(np.array([1.0, -1.0, 0.0]) / np.sqrt(2))),
    "line": ((-5, -5, 0.5), (5, 5, 0.5), (0, 0, 0)),
}


@pytest.mark.parametrize("name", list(PLANES))
def test_planes(name):
    p = abi.make_params(lam=2.2, condenser=(0, 0.5), objective=(0, 0.5), plane=PLANES[name], resolution=8, padding=1,
                        supersample=1, lut_us=False)
    s = [(0.5, 0.5, 0.5, 1.4, 1.4, 0.03), (-3.0, -2.5, 2.0, 1.1, 1.5, 0.0), (2.0, 4.0, 0.5, 0.7, 1.3, 0.01)]
    w = scenes.mc_waves(40, 0, 0.5, seed=31)
    U = oracle_lib.simulate(p, *abi.sphere_array(s), w)[0]
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.simulate(BS_PREC_FP64)
        err = np.linalg.norm(ctx.field() - U) / np.linalg.norm(U)
    assert err <= 1e-10, err
