"""The FP64 form's pair passes take four lanes to a particle, 64 (density) and 32 (force) particles to a block:
particle counts around those blocks and around one warp, from one particle on, against the oracle, through the
lists, the cell walk (lists overflow at the largest) and beside a second impact."""
import numpy as np
import pytest

from deorbit_gb300 import ic
from oracle import oracle as O

from parity import DERIV, STATE, field_errors, read_all

pytestmark = pytest.mark.gpu


def few(n):
    """The first n particles of a small impact with strength, in lattice order."""
    sc = ic.sized_impact(600, seed=5, angle_deg=30.0, speed=3000.0, ratio=0.3)
    sc.params.update(damage_on=0, flaw_model=0)
    sc.flaws = None
    full = sc.n
    for k, a in list(vars(sc).items()):
        if isinstance(a, np.ndarray) and a.ndim and a.shape[0] == full:
            setattr(sc, k, a[full - n:].copy())
    assert sc.n == n
    return sc


# The sums have the same terms in another order: rounding alone (1e-16 relative a term, terms that cancel to
# about 1e-4 of their size in the rates), far inside the parity bound of 1e-9.
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 129, 515])
@pytest.mark.parametrize("how", ["list", "cells", "beside"])
def test_sizes_match_oracle(cuda_lib, oracle_lib, n, how):
    from deorbit_gb300 import sph
    sc = few(n)
    ctx = sph.Context(sph.FP64)
    if how == "cells":  # far more neighbours than a list holds at first
        sc.params = dict(sc.params, eta=2.8, h_init=2.8 * sc.dx)
    ids = {}
    if how == "beside":
        ic.to_context(ctx, few(77), material_ids=ids)
    b = ic.to_context(ctx, sc, material_ids=ids)
    orc = O.from_scenario(sc)
    ctx.init()
    orc.init()
    for _ in range(2):
        dt = orc.timestep()
        assert abs(ctx.timestep(b) - dt) <= 1e-9 * dt
        orc.step(dt)
        ctx.step(dt)
    names = STATE + DERIV
    errs = field_errors(read_all(ctx, b, names), {k: orc.field(k) for k in names}, names)
    ctx.close()
    assert max(errs.values()) <= 1e-9, errs


@pytest.mark.parametrize("strength", [False, True])
def test_written_stress_matches_oracle(cuda_lib, oracle_lib, strength):
    """An impact without stress leaves the stress terms out of its force pass; one particle's stress, written
    between two steps, brings them back (and the written zeros take them out again)."""
    from deorbit_gb300 import sph
    sc = few(515)
    if not strength:
        sc.materials = [ic.granite(strength=False), ic.iron(strength=False)]
    ctx = sph.Context(sph.FP64)
    b = ic.to_context(ctx, sc)
    orc = O.from_scenario(sc)
    ctx.init()
    orc.init()
    names = [k for k in STATE + DERIV if strength or k not in ("dSxx", "dSyy", "dSzz", "dSxy", "dSxz", "dSyz")]
    for stress in (None, 3.0e8, 0.0):
        if stress is not None:
            for k in ("Sxx", "Sxy"):
                s = orc.field(k)
                s[:] = 0.0
                s[200] = stress
                orc.set_field(k, s)
                ctx.write(b, k, s)
        dt = orc.timestep()
        orc.step(dt)
        ctx.step(dt)
        errs = field_errors(read_all(ctx, b, names), {k: orc.field(k) for k in names}, names)
        assert max(errs.values()) <= 1e-9, (stress, errs)
    ctx.close()
