"""dmrg_env_step_order without a dual tensor: psi takes its place in psi's own order, whatever the
dual's order bit says. The reordered operands are the same numbers, so the results are the same."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DP = C.POINTER(C.c_double)


@pytest.mark.parametrize("left", [0, 1])
@pytest.mark.parametrize("bits", range(8))
def test_null_dual_is_psi(dmrgb, ctx, left, bits):
    ml, d, mr, w = 7, 2, 5, 3
    rng = np.random.default_rng(bits)
    A = rng.standard_normal((ml, d, mr))
    W = np.asfortranarray(rng.standard_normal((w, d, d, w)))
    m, k = (ml, mr) if left else (mr, ml)
    E = rng.standard_normal((m, w, m))
    ptr = lambda x: x.ctypes.data_as(DP)
    order = lambda x, rows: np.ascontiguousarray(x) if rows else np.asfortranarray(x)
    out = []
    for dual in (None, order(A, bits & 2)):
        res = np.full((k, w, k), np.nan, order="F")
        code = dmrgb.lib().dmrg_env_step_order(
            ctx.h, left, ml, d, mr, w, w, ptr(order(E, bits & 1)),
            None if dual is None else ptr(dual), ptr(order(A, bits & 2)), ptr(W), ptr(res),
            bits if dual is None else (bits & 3) | (4 if bits & 2 else 0))
        assert code == 0, dmrgb.lib().dmrg_last_error(ctx.h)
        out.append(res)
    assert np.array_equal(out[0], out[1])
