"""The double-precision LUT kernel's arc cosine over the whole angle range: a plane above and below a small
sphere (forward and backward directions through the poles), wide condensers, few and many table columns;
against the oracle at the parity suite's 1e-10."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_PREC_FP64, Context, abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z", [2.5, -2.5, 0.0])
@pytest.mark.parametrize("theta", [2, 37, 1000, 5000])
def test_angles(z, theta):
    p = abi.make_params(lam=2.5, condenser=(0, 1.0), objective=(0, 0.5), xy=(8, z), resolution=11, padding=1,
                        supersample=1, us_lut_r=60, us_lut_theta=theta)
    s = [(0.0, 0.0, 0.0, 1.0, 1.45, 0.03)]
    w = np.concatenate([scenes.mc_waves(60, 0, 1.0, seed=41), [[0, 0, 1.0], [0, 0, -1.0], [1.0, 0, 0]]])
    U = oracle_lib.simulate(p, *abi.sphere_array(s), w)[0]
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.simulate(BS_PREC_FP64)
        err = np.linalg.norm(ctx.field() - U) / np.linalg.norm(U)
    assert err <= 1e-10, err


def test_directions_that_are_not_unit_vectors():
    """Cosines beyond 1, up to and past the range of a float: the angle clamps at 0 and pi."""
    p = abi.make_params(lam=2.5, condenser=(0, 0.5), objective=(0, 0.5), xy=(8, 0), resolution=11, padding=1,
                        supersample=1, us_lut_r=60, us_lut_theta=90)
    s = [(0.0, 0.0, 0.0, 1.0, 1.45, 0.03)]
    scale = np.concatenate([np.linspace(0.8, 1.3, 56), [1e3, 1e30, 1e39, 1e60]])
    w = scenes.mc_waves(60, 0, 0.5, seed=43) * scale[:, None]
    U = oracle_lib.simulate(p, *abi.sphere_array(s), w)[0]
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.simulate(BS_PREC_FP64)
        err = np.linalg.norm(ctx.field() - U) / np.linalg.norm(U)
    assert err <= 1e-10, err
