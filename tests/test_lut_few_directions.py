"""No step in the time of a mixed slice where the directions pass 32: one more direction is 3 % more work.  Half as
much again leaves room for a second pass over the tile; ordering two groups of directions took 2.4 times."""
import pytest

from bimsim_gb300 import BS_PREC_MIXED, Context, abi, scenes

pytestmark = pytest.mark.gpu


def field_ms(nk):
    p = abi.make_params(lam=3.0, condenser=(0, 0.5), objective=(0, 0.5), xy=(60, 0), resolution=512, padding=1,
                        supersample=1)
    with Context(p) as ctx:
        ctx.set_spheres(scenes.random_spheres(20, 60.0, 0.9, 2.5, seed=5))
        ctx.set_waves(scenes.mc_waves(nk, 0, 0.5, seed=3))
        ms = []
        for _ in range(5):
            ctx.simulate(BS_PREC_MIXED)
            ms.append(ctx.stats().ms_us)
        return min(ms)


def test_33_directions_cost_about_as_much_as_32():
    a, b = field_ms(32), field_ms(33)
    assert b <= 1.5 * a, (a, b)
