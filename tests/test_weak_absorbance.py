"""Absorbance of slices with little contrast, in mixed precision, against the recorded images.

Such an image is the logarithm of a quotient near one of two float images, each 1e-7 off, and hangs on the order
and the number of the products between roundings.  The same arithmetic in the same order gives the same
image; 2e-6 leaves 30 roundings of a float for other double-precision instructions in what comes before.
Any other order of the sums moves these images by 5e-6 to 4e-5."""
import base64
import json
import os

import numpy as np
import pytest

from bimsim_gb300 import BS_IMG_ABSORBANCE, BS_PREC_MIXED, Context, abi, scenes

pytestmark = pytest.mark.gpu

with open(os.path.join(os.path.dirname(__file__), "golden", "weak_absorbance.json")) as _f:
    SCENES = json.load(_f)["scenes"]


def image(c):
    tables = c["method"] == "tables"
    p = abi.make_params(lam=c["lam"], condenser=(0, c["na"]), objective=(0, c["na"]), xy=tuple(c["xy"]),
                        resolution=c["resolution"], padding=1, supersample=1, lut_us=tables, lut_uf=tables)
    with Context(p) as ctx:
        ctx.set_spheres([tuple(s) for s in c["spheres"]])
        ctx.set_waves(scenes.mc_waves(c["waves"], 0, c["na"], seed=c["seed"]))
        ctx.simulate(BS_PREC_MIXED)
        return ctx.image(BS_IMG_ABSORBANCE)


@pytest.mark.parametrize("i", range(len(SCENES)))
def test_recorded_image(i):
    c = SCENES[i]
    a = image(c).astype(np.float64)
    b = np.frombuffer(base64.b64decode(c["absorbance"]), dtype="<f4").reshape(a.shape).astype(np.float64)
    assert np.linalg.norm(a - b) <= 2e-6 * np.linalg.norm(b), np.linalg.norm(a - b) / np.linalg.norm(b)
