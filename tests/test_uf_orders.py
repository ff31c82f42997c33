"""The incident-field kernels over the field order (even and odd counts, none, many), direct and from the table,
with the clamped orders (k d small) in the slice; double precision against the oracle (1e-10)."""
import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_FIELD_INCIDENT, BS_PREC_FP64, Context, abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lut_uf", [False, True])
@pytest.mark.parametrize("order", [0, 1, 2, 11, 60])
def test_orders(order, lut_uf):
    p = abi.make_params(lam=2.5, amplitude=1.7, focus=(0.25, -0.5, 0.0), condenser=(0.1, 0.6), objective=(0, 0.5),
                        xy=(12, 0), resolution=12, padding=1, field_order=order, lut_uf=lut_uf, uf_lut_r=90)
    w = scenes.mc_waves(8, 0.1, 0.6, seed=2)
    Uf = oracle_lib.simulate(p, *abi.sphere_array([]), w)[1]
    with Context(p) as ctx:
        ctx.set_spheres([])
        ctx.set_waves(w)
        ctx.simulate(BS_PREC_FP64)
        err = np.linalg.norm(ctx.field(BS_FIELD_INCIDENT) - Uf) / np.linalg.norm(Uf)
    assert err <= 1e-10, err
