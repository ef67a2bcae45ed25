"""Blocks of 1 to 40 states beside a larger one, which take the many-CTA eigensolver with it, after a
kernel that leaves NaN in the shared memory of every SM: no number may come from a word that the
solver has not written. Tolerances: an orthonormal vector of up to 400 rows carries about
sqrt(n) rounding units, 1e-13 bounds it, and the residual of a backward-stable solver n times the
rounding unit with a factor for its constant, 2e-14 ||A|| for the values and 1e-12 ||A|| for the
vectors."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DP = C.POINTER(C.c_double)


def _check(dmrgb, ctx, mats, ks):
    ns = [M.shape[0] for M in mats]
    A = np.concatenate([M.ravel() for M in mats])         # symmetric: the order does not matter
    w = np.full(sum(ns), np.nan)
    U = np.full(max(1, sum(n * k for n, k in zip(ns, ks))), np.nan)
    code = dmrgb.lib().dmrg_test_syevt_dirty(ctx.h, len(ns), (C.c_int * len(ns))(*ns),
                                             (C.c_int * len(ks))(*ks), A.ctypes.data_as(DP),
                                             w.ctypes.data_as(DP), U.ctypes.data_as(DP))
    assert code == 0, dmrgb.lib().dmrg_last_error(ctx.h)
    ow = ou = 0
    for M, n, k in zip(mats, ns, ks):
        lam, V = w[ow:ow + n], U[ou:ou + n * k].reshape((n, k), order="F")
        nrm = np.linalg.norm(M, 2)
        assert np.all(np.isfinite(lam)) and np.all(np.isfinite(V)), (n, k)
        assert np.max(np.abs(lam - np.linalg.eigvalsh(M)[::-1])) <= 2e-14 * nrm, (n, k)
        if k:
            assert np.max(np.abs(V.T @ V - np.eye(k))) <= 1e-13, (n, k)
            assert np.max(np.abs(M @ V - V * lam[:k])) <= 1e-12 * nrm, (n, k)
        ow += n
        ou += n * k


@pytest.mark.parametrize("large", [41, 120, 300, 400, 600])
@pytest.mark.parametrize("kept", ["all", "half", "one"])
def test_small_blocks_beside_a_large_one(dmrgb, ctx, large, kept):
    rng = np.random.default_rng(large)
    mats = []
    for n in [large, *range(1, 41)]:
        Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        M = (Q * 10.0 ** (-np.arange(n) * 8.0 / n)) @ Q.T
        mats.append(0.5 * (M + M.T))
    ks = [{"all": n, "half": (n + 1) // 2, "one": 1}[kept] for n in (M.shape[0] for M in mats)]
    ks[0] = min(ks[0], 200)
    _check(dmrgb, ctx, mats, ks)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 8, 15, 31, 32, 33, 39, 40])
def test_small_blocks_alone(dmrgb, ctx, n):
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n))
    _check(dmrgb, ctx, [M @ M.T / n] * 2, [n, (n + 1) // 2])
