"""Both tile shapes of the grouped FP64 GEMM at every size, leading dimension and transpose: a context
of its own per case, so that its first calls try both (the choice of a session's context is made by
block-size class, and later sizes of a class would run one shape only). Bounds as in
test_gpu_gemm.py: 2.1 K u relative to sum_k |a_ik||b_kj|; the shapes agree bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DP = C.POINTER(C.c_double)


@pytest.mark.parametrize("tA,tB", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 3), (31, 15, 31), (32, 16, 32), (33, 17, 33), (32, 32, 64),
                                   (47, 33, 95), (64, 48, 97), (100, 100, 500)])
@pytest.mark.parametrize("pad", [0, 1])
def test_both_shapes_run_and_agree(dmrgb, tA, tB, M, N, K, pad):
    rng = np.random.default_rng(M + 3 * N + 5 * K + pad)
    A = np.asfortranarray(rng.standard_normal(((K if tA else M) + pad, M if tA else K)))
    B = np.asfortranarray(rng.standard_normal(((N if tB else K) + pad, K if tB else N)))
    a, b = A[:K if tA else M], B[:N if tB else K]
    a, b = (a.T if tA else a), (b.T if tB else b)
    own = dmrgb.Context(0)
    runs = []
    for _ in range(12):
        out = np.asfortranarray(np.full((M + pad, N), np.nan))
        code = dmrgb.lib().dmrg_test_gemm(own.h, tA, tB, M, N, K, A.ctypes.data_as(DP), A.shape[0],
                                          B.ctypes.data_as(DP), B.shape[0],
                                          out.ctypes.data_as(DP), M + pad)
        assert code == 0, dmrgb.lib().dmrg_last_error(own.h)
        runs.append(out)
    assert own.tuner()[:2] == (1, 1)       # one class of sizes, decided: both shapes were timed
    assert np.all(np.abs(runs[0][:M] - a @ b) <= 2.1 * K * 2.0 ** -53 * (np.abs(a) @ np.abs(b)))
    for r in runs[1:]:
        assert np.array_equal(r[:M], runs[0][:M])
    assert np.all(np.isnan(runs[0][M:]))
