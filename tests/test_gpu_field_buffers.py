"""Several fields in one call: page-locked buffers are reached by the kernels themselves, others through the staging
buffer.  Both, mixed in one call, buffers off their natural alignment and more fields than one launch takes must
carry the same numbers, in either direction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("x y z vx vy vz u hh ax ay az dudt Sxx Syy Szz Sxy Sxz Syz dSxx").split()


@pytest.mark.parametrize("precision", [0, 1])
def test_buffers_carry_the_same_fields(cuda_lib, precision):
    import ctypes

    import torch
    from deorbit_gb300 import ic, sph
    L = sph.lib()
    ctx = sph.Context(precision)
    ids = {}
    bs = [ic.to_context(ctx, ic.sized_impact(n, seed=n, angle_deg=40.0, speed=9000.0, ratio=0.25), material_ids=ids)
          for n in (700, 3000)]
    ctx.init()
    ctx.run(2)
    for b in bs:
        n = ctx.n(b)
        want = {k: ctx.read(b, k) for k in NAMES}

        def buffers(kind):
            out = []
            for i, _ in enumerate(NAMES):
                pinned = kind in ("pinned", "odd") or (kind == "mixed" and i % 2 == 1)
                raw = torch.empty(8 * n + 16, dtype=torch.uint8, pin_memory=pinned).numpy()
                out.append((raw, raw.ctypes.data + (4 if kind == "odd" and i % 3 == 0 else 0)))
            return out

        cn = (ctypes.c_char_p * len(NAMES))(*[k.encode() for k in NAMES])
        for kind in ("pinned", "pageable", "mixed", "odd"):
            bufs = buffers(kind)
            ptrs = (ctypes.POINTER(ctypes.c_double) * len(NAMES))(
                *[ctypes.cast(a, ctypes.POINTER(ctypes.c_double)) for _, a in bufs])
            sph.check(L.sph_read_fields(ctx.h, b, len(NAMES), cn, ptrs))
            for k, (raw, a) in zip(NAMES, bufs):
                off = a - raw.ctypes.data
                assert raw[off:off + 8 * n].tobytes() == want[k].tobytes(), (kind, k)
            for k in NAMES:  # other values in, then these back
                ctx.write(b, k, want[k] + 1.0)
            sph.check(L.sph_write_fields(ctx.h, b, len(NAMES), cn, ptrs))
            for k in NAMES:
                assert np.array_equal(ctx.read(b, k), want[k]), (kind, k)
    ctx.close()
