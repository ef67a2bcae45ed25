"""The grouped FP64 GEMM around its tile and slice sizes (32 x 32 and 32 x 16 tiles, slices of 32
in K, a ring of four), with even and odd leading dimensions (16- and 8-byte copies) and all
transposes. An element is one chain of K fused multiply-adds, so it lies within K u / (1 - K u) of
the exact value relative to sum_k |a_ik||b_kj| (u = 2^-53), numpy's product within the same bound:
2.1 K u in all. Both tile shapes sum in the same order, so they agree bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DP = C.POINTER(C.c_double)


def _run(dmrgb, ctx, tA, tB, A, B, M, N, K, ldc):
    out = np.asfortranarray(np.full((ldc, N), np.nan))
    code = dmrgb.lib().dmrg_test_gemm(ctx.h, tA, tB, M, N, K, A.ctypes.data_as(DP), A.shape[0],
                                      B.ctypes.data_as(DP), B.shape[0], out.ctypes.data_as(DP),
                                      ldc)
    assert code == 0, dmrgb.lib().dmrg_last_error(ctx.h)
    return out


@pytest.mark.parametrize("tA,tB", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 3), (8, 8, 4), (31, 15, 31), (32, 16, 32), (33, 17, 33),
                                   (32, 32, 64), (47, 33, 95), (64, 48, 97), (100, 100, 500),
                                   (1500, 700, 130)])
@pytest.mark.parametrize("pad", [0, 1])
def test_tiles_and_slices(dmrgb, ctx, tA, tB, M, N, K, pad):
    rng = np.random.default_rng(M + 3 * N + 5 * K + pad)
    A = np.asfortranarray(rng.standard_normal(((K if tA else M) + pad, M if tA else K)))
    B = np.asfortranarray(rng.standard_normal(((N if tB else K) + pad, K if tB else N)))
    a, b = A[:K if tA else M], B[:N if tB else K]
    a, b = (a.T if tA else a), (b.T if tB else b)
    runs = [_run(dmrgb, ctx, tA, tB, A, B, M, N, K, M + pad) for _ in range(4)]
    bound = 2.1 * K * 2.0 ** -53 * (np.abs(a) @ np.abs(b))
    assert np.all(np.abs(runs[0][:M] - a @ b) <= bound)
    for r in runs[1:]:                     # both tile shapes are on trial in the first calls
        assert np.array_equal(r[:M], runs[0][:M])
    assert np.all(np.isnan(runs[0][M:]))   # rows between M and the leading dimension stay
