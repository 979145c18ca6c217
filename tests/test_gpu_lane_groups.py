"""Runs of few particles take eight lanes to a particle in the list build and the pair passes; larger ones a
thread.  An impact must give the same bits either way: alone (lanes) and beside one that lifts the context past
the changeover (threads)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x y z vx vy vz u rho hh P D ax ay az dudt Sxx Syy Szz Sxy Sxz Syz dSxx dSyy dSzz dSxy dSxz dSyz").split()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,slack", [(1000, 0.03), (1777, 1e-7), (6000, 0.03), (20000, 1e-7)])
def test_lanes_equal_threads(cuda_lib, precision, n, slack):
    from deorbit_gb300 import ic, sph
    sc = ic.sized_impact(n, seed=n, angle_deg=40.0, speed=9000.0, ratio=0.25)
    filler = ic.sized_impact(70000, seed=3, angle_deg=20.0, speed=6000.0, ratio=0.2, strength=False)
    got = []
    for scs in ([sc], [sc, filler]):
        ctx = sph.Context(precision)
        ctx.set_option("slack", slack)  # a tiny slack sends particles whose h grows to the refresh and the fallback
        ids = {}
        bs = [ic.to_context(ctx, s, material_ids=ids) for s in scs]
        ctx.init()
        ctx.run(5)
        ctx.step(ctx.timestep(bs[0]))
        got.append({k: ctx.read(bs[0], k) for k in FIELDS})
        ctx.close()
    for k in FIELDS:
        assert np.array_equal(got[0][k], got[1][k]), k
        assert np.isfinite(got[0][k]).all(), k
