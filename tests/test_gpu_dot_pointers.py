"""fmg_dot_noalloc on a caller's own pointers: any address a double may have,
so also the odd ones of a slice, at lengths around a pair and a chunk -- equal
to the oracle's reduction of the same values (one order on both sides)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ox,oy", [(0, 0), (1, 0), (0, 1), (1, 1), (2, 3)])
def test_dot_noalloc_of_slices(oracle_mod, ox, oy):
    import torch

    import gnu_femlisp_b200 as G
    ctx = G.Context(0)
    lib = G._capi.load()
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    for n in (1, 2, 511, 4095, 4096, 4097, 3 * 4096 + 2, 592 * 4096, 592 * 4096 + 3):  # the last: more than a wave
        rng = np.random.default_rng(10 * n + ox)
        x, y = rng.standard_normal(n + 4), rng.standard_normal(n + 4)
        xd, yd = torch.from_numpy(x).to("cuda"), torch.from_numpy(y).to("cuda")
        torch.cuda.synchronize()
        ctx.check(lib.fmg_dot_noalloc(ctx.h, ctypes.c_void_p(xd.data_ptr() + 8 * ox),
                                      ctypes.c_void_p(yd.data_ptr() + 8 * oy), n, ctypes.c_void_p(out.data_ptr())),
                  "fmg_dot_noalloc")
        ctx.synchronize()
        assert float(out.item()) == oracle_mod.dot(x[ox:ox + n], y[oy:oy + n]), n
