"""Dense operands on their way to the device and back: memory orders of the environment step's
operands, and environments and vectors longer than one piece of the staging (1 MB).

The orders only change how an operand is copied, so the results are the same bits. Against numpy:
an element of an environment step is a sum of at most w d m^2 products in three nested
contractions, each of K terms within K u relative to the sum of magnitudes (u = 2^-53)."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stored(x, how):
    if how == "F":
        return np.asfortranarray(x)
    if how == "C":
        return np.ascontiguousarray(x)
    big = np.zeros(tuple(2 * n for n in x.shape))        # neither
    big[::2, ::2, ::2] = x
    return big[::2, ::2, ::2]


@pytest.mark.parametrize("ml,mr,d,w", [(1, 1, 2, 1), (7, 33, 3, 5), (150, 211, 2, 5)])
@pytest.mark.parametrize("left", [True, False])
def test_orders_of_the_environment_step(dmrgb, ctx, ml, mr, d, w, left):
    rng = np.random.default_rng(ml + mr)
    A, D = rng.standard_normal((2, ml, d, mr))
    W = rng.standard_normal((w, d, d, w))
    m = ml if left else mr
    E = rng.standard_normal((m, w, m))
    f = dmrgb.Lupdate if left else dmrgb.Rupdate
    spec = "awb,wstv,bsd,atc->cvd" if left else "dvc,wstv,bsd,atc->bwa"
    path = ["einsum_path", (0, 2), (0, 2), (0, 1)]
    ref = np.einsum(spec, E, W, A, D, optimize=path)
    mag = np.einsum(spec, abs(E), abs(W), abs(A), abs(D), optimize=path)
    first = f(E, D, A, W, ctx=ctx)
    K = m + w * d + max(ml, mr) * d
    assert np.all(abs(first - ref) <= 2.5 * K * 2.0 ** -53 * mag)
    for e, p, q in itertools.product("FCN", repeat=3):
        assert np.array_equal(f(_stored(E, e), _stored(D, q), _stored(A, p), W, ctx=ctx), first)
    same = f(E, A, A, W, ctx=ctx)                        # one tensor for both
    assert np.array_equal(f(E, A.copy(order="F"), A, W, ctx=ctx), same)


def test_environments_and_vectors_of_many_pieces(dmrgb, ctx):
    """A dense state of 320 states: its environments (4.1 MB) and two-site vectors (3.3 MB)."""
    L, m = 18, 320
    rng = np.random.default_rng(3)
    dims = [min(2 ** i, 2 ** (L - i), m) for i in range(L + 1)]
    sites = [rng.standard_normal((dims[i], 2, dims[i + 1])) / np.sqrt(2 * dims[i + 1])
             for i in range(L)]
    mpo = dmrgb.makeMPO(dmrgb.heisenbergMPO, 2, L)
    psi = dmrgb.MPS(sites, oc=L // 2)
    Lenv, Renv = dmrgb.makeEnv(psi, mpo, ctx=ctx)
    i = L // 2
    dev = psi._dev
    for k in range(i, i + 2):                            # the next environments from these
        if k > i:
            dmrgb.Lupdate(k - 1, Lenv)
    nxt = dmrgb.Lupdate(Lenv[i], sites[i], sites[i], mpo.W[i], ctx=ctx)
    assert np.max(abs(Lenv[i + 1] - nxt)) <= 1e-12 * np.max(abs(nxt))
    x = rng.standard_normal((dims[i], 2, 2, dims[i + 2]))
    y = dev.heff(i, x)
    z = np.einsum("awb,wstv,vuxz,dzc,bsud->atxc", Lenv[i], mpo.W[i],
                  mpo.W[i + 1], Renv[i + 1], x,
                  optimize=["einsum_path", (0, 4), (0, 3), (0, 2), (0, 1)])
    assert np.max(abs(y - z)) <= 1e-12 * np.max(abs(z))
