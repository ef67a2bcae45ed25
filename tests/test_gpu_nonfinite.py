"""A state or an operator that holds a NaN or an infinity ends a solve at the bond step that meets it,
with an error, in every kind of solve; the context solves the next problem as ever."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(dmrgb, ctx, kind, psi, mpo, krylov, precision="fp64"):
    if kind == "tdvp":
        dmrgb.tdvp_twosite(psi, mpo, m=24, cutoff=1e-10, r=krylov, prefactor=-1.0,
                           precision=precision, ctx=ctx)
    else:
        dmrgb.dmrg(psi, mpo, m=24, sweeps=1, cutoff=1e-10, krylov=krylov, precision=precision,
                   method="3S" if kind == "3s" else "twosite", ctx=ctx)


@pytest.mark.parametrize("kind", ["twosite", "3s", "tdvp"])
@pytest.mark.parametrize("krylov,precision", [(2, "fp64"), (4, "fp64"), (4, "3xtf32")])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("where", ["state", "operator"])
def test_nonfinite_input_is_an_error(dmrgb, ctx, kind, krylov, precision, value, where):
    L = 8
    mpo = dmrgb.makeMPO(dmrgb.heisenbergMPO, 2, L)
    psi = dmrgb.randMPS(2, L, 24, seed=1)
    if where == "state":
        psi.tensors[L // 2][1, 0, 1] = value
    else:
        mpo.W[L // 2][-1, 0, 0, 0] = value
    with pytest.raises(dmrgb.DmrgError, match="not finite"):
        _solve(dmrgb, ctx, kind, psi, mpo, krylov, precision)
    good = dmrgb.randMPS(2, L, 24, seed=2)
    _solve(dmrgb, ctx, kind, good, dmrgb.makeMPO(dmrgb.heisenbergMPO, 2, L), krylov, precision)
    assert np.isfinite(good.sweep_stats[-1]["energy"])


@pytest.mark.parametrize("n", [41, 200, 600])
def test_eigenvalues_of_a_nonfinite_block_are_no_numbers(dmrgb, ctx, n):
    import ctypes as C
    dp = C.POINTER(C.c_double)
    A = np.eye(n)
    A[n // 2, n // 2] = np.nan
    w, U = np.zeros(n), np.zeros(n)
    assert dmrgb.lib().dmrg_test_syevt(ctx.h, 1, (C.c_int * 1)(n), (C.c_int * 1)(0),
                                       A.ctypes.data_as(dp), w.ctypes.data_as(dp),
                                       U.ctypes.data_as(dp)) == 0
    assert np.all(np.isnan(w))
