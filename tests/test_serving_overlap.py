"""A short request on a fresh context finishes while a long one runs: no call of the long one's thread may hold up
the other threads' calls while its kernels run."""
import time

import pytest

from bimsim_gb300 import BS_IMG_INTENSITY, BS_PREC_MIXED, Server, abi, scenes

pytestmark = pytest.mark.gpu


def request(res, ns, nk):
    p = abi.make_params(lam=4.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(100, 0), resolution=res, padding=1,
                        lut_uf=True, us_lut_r=1024, us_lut_theta=1024, uf_lut_r=256, supersample=1)
    return p, scenes.random_spheres(ns, 100.0, 0.5, 1.5, seed=71), scenes.mc_waves(nk, 0.0, 0.5, seed=72)


def test_short_request_beside_a_long_one():
    # 1.9e12 lookups, above two seconds of the GPU, against 1e8
    (p, s, w), (q, t, v) = request(768, 180, 2000), request(64, 10, 200)
    with Server(workers=2) as srv:
        long = srv.submit(p, s, waves=w, precision=BS_PREC_MIXED, image=BS_IMG_INTENSITY)
        time.sleep(0.5)
        short = srv.submit(q, t, waves=v, precision=BS_PREC_MIXED, image=BS_IMG_INTENSITY)
        srv.wait(short, 60.0)
        running = not srv.poll(long)
        srv.wait(long, 120.0)
        assert srv.stats().failed == 0
    assert running
