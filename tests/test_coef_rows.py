"""Coefficient rows of the table paths: orders up to the largest the library accepts (512), blocks whose rows belong to
several spheres, and contexts of different orders on several threads, against the oracle.  Double-precision
results to the parity suite's 1e-10; a float table entry is within half an ulp, 6e-8 of the largest entry
bounds every one and 2e-7 leaves room for the build."""
import threading

import numpy as np
import pytest

import oracle_lib
from bimsim_gb300 import BS_IMG_INTENSITY, BS_PREC_FP64, BS_PREC_MIXED, Context, abi, scenes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def filler(n):
    """Small spheres off to one side: more than 8 in all select the sorted kernel and its tables."""
    return [(-3.5 + 0.8 * i, 3.6, 0.0, 0.3, 1.3, 0.0) for i in range(n)]


# one sphere of 11 orders with a field order whose count of orders passes 435, the most of a block's shared memory
@pytest.mark.parametrize("order", [100, 434, 435, 512])
@pytest.mark.parametrize("extra", [0, 8])
def test_high_field_orders(order, extra):
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(10, 0), resolution=8, padding=1,
                        us_lut_r=40, us_lut_theta=200, field_order=order)
    s = [(1.0, -0.5, 0.0, 1.5, 1.4, 0.02)] + filler(extra)
    w = scenes.mc_waves(70, 0, 0.5, seed=4)
    U, _, D, _ = oracle_lib.simulate(p, *abi.sphere_array(s), w)
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(w)
        ctx.simulate(BS_PREC_FP64)
        assert rel(ctx.field(), U) <= 1e-10
        ctx.simulate(BS_PREC_MIXED)
        assert rel(ctx.image(BS_IMG_INTENSITY, f64=True), D) <= 1e-5


def tables_agree(ctx, p, s, tol, which_spheres=None):
    lib = oracle_lib.load()
    for i, sp in enumerate(s):
        if which_spheres is not None and i not in which_spheres:
            continue
        g = oracle_lib.sphere_geom(p, abi.Sphere(*sp))
        ref = [np.zeros(2 * g.dR * g.thetaR), np.zeros(2 * g.aR * g.thetaR)]
        lib.bso_sphere_luts(oracle_lib.C.byref(p), oracle_lib.C.byref(abi.Sphere(*sp)), oracle_lib.P(ref[0]),
                            oracle_lib.P(ref[1]))
        for which, n in ((0, g.dR), (1, g.aR)):
            r = ref[which].view(np.complex128).reshape(n, g.thetaR)
            t = ctx.lut(i, which, n, g.thetaR)
            for row in range(n):
                assert np.abs(t[row] - r[row]).max() <= tol * np.abs(r[row]).max(), (i, which, row)


# spheres of 421, 437 and 505 orders; alone and beside more than 8 small ones
@pytest.mark.parametrize("a", [62.0, 64.5, 75.0])
@pytest.mark.parametrize("extra", [0, 8])
def test_tables_of_large_spheres(a, extra):
    p = abi.make_params(lam=1.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(10, 0), resolution=8, padding=1,
                        us_lut_r=12, us_lut_theta=50)
    s = [(0.0, 0.0, a + 1.0, a, 1.02, 0.0)] + filler(extra)
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(scenes.mc_waves(70, 0, 0.5, seed=3))
        for prec, tol in ((BS_PREC_FP64, 1e-10), (BS_PREC_MIXED, 2e-7)):
            ctx.simulate(prec)
            tables_agree(ctx, p, s, tol, {0})


# eight and nine spheres whose inner rows share blocks with other spheres' outer rows: every row of every table
@pytest.mark.parametrize("seed", [16, 21])
@pytest.mark.parametrize("ns", [8, 9])
def test_every_row_of_many_spheres(seed, ns):
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(24, 0), resolution=96, padding=1,
                        supersample=1, us_lut_theta=60)
    s = scenes.random_spheres(8, 24.0, 0.8, 2.5, seed=seed * 1009 + 2, z_slab=0.0)
    s = list(s) + [(11.0, 11.0, 0.0, 0.7, 1.3, 0.0)] * (ns - 8)
    with Context(p) as ctx:
        ctx.set_spheres(s)
        ctx.set_waves(scenes.mc_waves(70, 0, 0.5, seed=seed))
        for prec, tol in ((BS_PREC_FP64, 1e-10), (BS_PREC_MIXED, 2e-7)):
            ctx.simulate(prec)
            tables_agree(ctx, p, s, tol)


def test_contexts_of_different_orders_at_once():
    """Two threads, slices of 109 and of 298 orders in turn: every one runs and gives its own result."""
    scene = []
    for a in (14.0, 43.0):
        p = abi.make_params(lam=1.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(10, 0), resolution=8, padding=1,
                            us_lut_r=12, us_lut_theta=50)
        scene.append((p, [(0.0, 0.0, a + 1.0, a, 1.02, 0.0)], scenes.mc_waves(20, 0, 0.5, seed=3)))
    want, failed = [], []
    for p, s, w in scene:
        with Context(p) as ctx:
            ctx.set_spheres(s)
            ctx.set_waves(w)
            ctx.simulate(BS_PREC_FP64)
            want.append(ctx.field())

    def loop(k):
        try:
            p, s, w = scene[k]
            with Context(p) as ctx:
                ctx.set_spheres(s)
                ctx.set_waves(w)
                for _ in range(200):
                    ctx.simulate(BS_PREC_FP64)
                    assert np.array_equal(ctx.field(), want[k])
        except BaseException as e:  # noqa: B036
            failed.append(repr(e))

    threads = [threading.Thread(target=loop, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
