"""A kernel's limit of dynamic shared memory belongs to the kernel on the device, for all threads of the process: a call
that sets it to its own size lets another context's launch fail.  Every setting is to a constant."""
import glob
import os
import re
import threading

import numpy as np
import pytest

from bimsim_gb300 import BS_PREC_FP64, Context, abi, scenes

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bimsim-cuda_gb300", "csrc")


def test_limits_are_constants():
    sizes, constants = [], set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.h")):
        text = open(path).read()
        sizes += re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*([^;]+)\);", text)
        constants |= set(re.findall(r"constexpr int (\w+) =", text))
    assert sizes and all(s in constants for s in sizes), sizes


@pytest.mark.gpu
def test_direct_slices_of_different_orders_at_once():
    """Two threads, direct slices of 57 and of 187 orders in turn (57 and 187 KB a block)."""
    scene = []
    for a in (6.5, 26.0):
        p = abi.make_params(lam=1.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(10, 0), resolution=4, padding=1,
                            lut_us=False, lut_uf=False)
        scene.append((p, [(0.0, 0.0, a + 1.0, a, 1.02, 0.0)], scenes.mc_waves(8, 0, 0.5, seed=3)))
    want, failed = [None, None], []

    def loop(k, n):
        try:
            p, s, w = scene[k]
            with Context(p) as ctx:
                ctx.set_spheres(s)
                ctx.set_waves(w)
                for _ in range(n):
                    ctx.simulate(BS_PREC_FP64)
                    f = ctx.field()
                    assert want[k] is None or np.array_equal(f, want[k])
                    want[k] = f
        except BaseException as e:  # noqa: B036
            failed.append(repr(e))

    loop(0, 1)
    loop(1, 1)
    threads = [threading.Thread(target=loop, args=(k, 200)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
