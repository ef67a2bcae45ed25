"""The one-launch Krylov vector kernel against the general launches, bit for bit: both sum every dot
product in the same order, so that the line between them (KRY_MAX elements) changes no number.
Vector lengths on either side of each count of elements per thread and of the summation blocks, all
modes, all iterations; a last block of the sums that is nearly empty, and a breakdown."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DP = C.POINTER(C.c_double)
NORMALISE, FIRST, STEP, ALPHA, LAST2 = range(5)
KK, KH, EN, COEF, A, B2, BETA, ACT = 16, 17, 19, 32, 48, 64, 80, 96
SIZES = [1, 2, 255, 256, 257, 8191, 8192, 8193, 16384, 16385, 32768, 32769, 40000, 65535, 65536]


def _run(dmrgb, ctx, general, mode, n, j, betatest, K, H, s):
    K, H, s = K.copy(), H.copy(), s.copy()
    code = dmrgb.lib().dmrg_test_krylov(ctx.h, general, mode, n, j, betatest, K.ctypes.data_as(DP),
                                        H.ctypes.data_as(DP), s.ctypes.data_as(DP))
    assert code == 0, dmrgb.lib().dmrg_last_error(ctx.h)
    return K, H, s


def _same(dmrgb, ctx, mode, n, j, slots, seed, betatest=1e-10, wreck=False, h_too=False):
    rng = np.random.default_rng(seed)
    K = rng.standard_normal((j + 2) * n) / np.sqrt(n)
    H = np.zeros(n) if wreck else rng.standard_normal(n)
    s = np.zeros(256)
    s[A:A + 16], s[BETA:BETA + 16], s[ACT:ACT + 17] = rng.standard_normal(16), rng.random(16), 1.0
    one = _run(dmrgb, ctx, 0, mode, n, j, betatest, K, H, s)
    all_ = _run(dmrgb, ctx, 1, mode, n, j, betatest, K, H, s)
    assert np.array_equal(one[0], all_[0], equal_nan=True)
    assert np.array_equal(one[2][slots], all_[2][slots], equal_nan=True)
    if h_too:
        assert np.array_equal(one[1], all_[1], equal_nan=True)
    return one


@pytest.mark.parametrize("n", SIZES)
def test_normalise_and_two_vector_step(dmrgb, ctx, n):
    _same(dmrgb, ctx, NORMALISE, n, 0, [0], n)
    _same(dmrgb, ctx, FIRST, n, 0, [KK, KH, A, B2, BETA, ACT + 1], n + 1)
    for seed in range(8):                  # the Ritz rotation's own roundings
        _same(dmrgb, ctx, LAST2, n, 1, [A + 1, EN, COEF, COEF + 1], n + 2 + seed, h_too=True)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("j", [0, 1, 2, 3, 6, 7, 14])
def test_lanczos_iterations(dmrgb, ctx, n, j):
    _same(dmrgb, ctx, STEP, n, j, [A + j, B2 + j, BETA + j, ACT + j + 1], n + j)
    _same(dmrgb, ctx, ALPHA, n, j, [A + j], n + j + 1)


@pytest.mark.parametrize("n", [1, 300, 8193, 65536])
def test_breakdown(dmrgb, ctx, n):
    K, _, s = _same(dmrgb, ctx, STEP, n, 2, [B2 + 2, BETA + 2, ACT + 3], n, betatest=1e30)
    assert s[BETA + 2] == 0.0 and s[ACT + 3] == 0.0 and not K[3 * n:].any()
    _same(dmrgb, ctx, STEP, n, 0, [A, B2, BETA, ACT + 1], n, wreck=True)
