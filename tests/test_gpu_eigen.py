"""Mid-size density-matrix blocks at the edges of the eigensolver's size classes (the clusters'
row and column capacities, the many-block rule), against numpy. Tolerances as for the other
eigensolver tests: the backward error of a Householder tridiagonalisation, n times the rounding
unit with a factor for its constant, is below 2e-14 ||A|| for n <= 512 and n/512 times that above;
orthonormality 1e-13 and residual 1e-12 ||A|| are what the truncation needs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DP = C.POINTER(C.c_double)


def _block(rng, n, kind):
    if kind == "graded":
        w = 10.0 ** (-np.arange(n) * 14.0 / n)
    elif kind == "pairs":                  # equal pairs, as spin multiplets give
        w = np.repeat(np.exp(-0.1 * np.arange((n + 1) // 2)), 2)[:n]
    elif kind == "rank1":
        w = np.zeros(n)
        w[0] = 1.0
    else:
        w = rng.uniform(0.1, 1.0, n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * w) @ Q.T
    return 0.5 * (A + A.T)


def _solve(dmrgb, ctx, mats, ks):
    ns = [M.shape[0] for M in mats]
    A = np.concatenate([np.asfortranarray(M).ravel(order="F") for M in mats])
    w = np.zeros(sum(ns))
    U = np.zeros(max(1, sum(n * k for n, k in zip(ns, ks))))
    code = dmrgb.lib().dmrg_test_syevt(ctx.h, len(ns), (C.c_int * len(ns))(*ns),
                                       (C.c_int * len(ks))(*ks), A.ctypes.data_as(DP),
                                       w.ctypes.data_as(DP), U.ctypes.data_as(DP))
    assert code == 0, dmrgb.lib().dmrg_last_error(ctx.h)
    ow = ou = 0
    for M, n, k in zip(mats, ns, ks):
        lam, Uk = w[ow:ow + n], U[ou:ou + n * k].reshape((n, k), order="F")
        nrm = np.linalg.norm(M, 2)
        assert np.max(np.abs(lam - np.sort(np.linalg.eigvalsh(M))[::-1])) < 2e-14 * max(1, n / 512) * nrm
        if k:
            assert np.max(np.abs(Uk.T @ Uk - np.eye(k))) < 1e-13
            assert np.max(np.abs(M @ Uk - Uk * lam[:k])) < 1e-12 * nrm
        ow += n
        ou += n * k


@pytest.mark.parametrize("n", [113, 160, 161, 224, 225, 256, 257, 320, 321, 352, 353, 448, 449, 512])
def test_block_size_edges(dmrgb, ctx, n):
    rng = np.random.default_rng(n)
    _solve(dmrgb, ctx, [_block(rng, n, "graded"), _block(rng, n, "flat")], [n // 2, n])


@pytest.mark.parametrize("n,k", [(513, 200), (544, 544), (545, 100), (1024, 512), (1025, 300),
                                 (2048, 150)])
def test_blocks_that_start_in_global_memory(dmrgb, ctx, n, k):
    """Above 512 rows the leading steps run on the matrix in global memory; smaller blocks in the
    same launches do not."""
    rng = np.random.default_rng(n)
    _solve(dmrgb, ctx, [_block(rng, n, "flat"), _block(rng, 150, "graded")], [k, 70])


@pytest.mark.parametrize("kind", ["pairs", "rank1"])
def test_degenerate_blocks(dmrgb, ctx, kind):
    rng = np.random.default_rng(7)
    ns = [120, 250, 400, 700]
    _solve(dmrgb, ctx, [_block(rng, n, kind) for n in ns], [60, 100, 150, 200])


@pytest.mark.parametrize("n", [260, 352])
def test_more_blocks_than_wide_clusters(dmrgb, ctx, n):
    """More than eight blocks take the eight-CTA clusters; sizes mixed, small blocks among them."""
    rng = np.random.default_rng(n + 1)
    ns = [n, n - 1, 300, 240, 200, 180, 170, 150, 140, 130, 120, 114, 90, 30, 3]
    _solve(dmrgb, ctx, [_block(rng, m, "graded") for m in ns], [m // 3 for m in ns])
