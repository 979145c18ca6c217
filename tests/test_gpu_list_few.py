"""Runs of few particles build their lists with a warp to a particle, larger ones with a thread to a particle.
An impact must give the same bits either way: alone (warps) and beside one that lifts the context past the
changeover (threads).  Sizes: from one particle on, boxes of more and of fewer columns than a warp has lanes (the
smoothing lengths), chords of many candidates, and lists that overflow."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x y z vx vy vz u rho hh P ax ay az dudt Sxx Syy Szz Sxy Sxz Syz").split()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,eta", [(1, 1.3), (3, 1.3), (65, 1.3), (65, 2.6), (1777, 1.3), (1777, 2.2), (20000, 1.3)])
def test_warps_equal_threads(cuda_lib, precision, n, eta):
    from deorbit_gb300 import ic, sph
    sc = ic.sized_impact(max(n, 600), seed=n, angle_deg=40.0, speed=9000.0, ratio=0.25)
    sc.params.update(damage_on=0, flaw_model=0, eta=eta, h_init=eta * sc.dx)
    sc.flaws = None
    if n < 600:
        full = sc.n
        for k, a in list(vars(sc).items()):
            if isinstance(a, np.ndarray) and a.ndim and a.shape[0] == full:
                setattr(sc, k, a[full - n:].copy())
    filler = ic.sized_impact(130000, seed=3, angle_deg=20.0, speed=6000.0, ratio=0.2, strength=False)
    got = []
    for scs in ([sc], [sc, filler]):
        ctx = sph.Context(precision)
        ids = {}
        bs = [ic.to_context(ctx, s, material_ids=ids) for s in scs]
        assert (sum(s.n for s in scs) > 90112) == (len(scs) == 2)
        ctx.init()
        ctx.run(3)
        ctx.step(ctx.timestep(bs[0]))
        got.append({k: ctx.read(bs[0], k) for k in FIELDS})
        ctx.close()
    for k in FIELDS:
        assert np.array_equal(got[0][k], got[1][k]), k
        assert np.isfinite(got[0][k]).all(), k
