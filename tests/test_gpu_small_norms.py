"""Density-matrix blocks whose norm is far from 1 (sectors of small weight), and Krylov matrices of
operators whose norm is: the Sturm counts multiply up to twelve numbers of that size. Tolerances are
those of the same solves at norm 1, relative to the block's own norm."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DP = C.POINTER(C.c_double)


def _values(dmrgb, ctx, M):
    n = M.shape[0]
    A, w, U = M.copy(), np.zeros(n), np.zeros((n, n), order="F")
    code = dmrgb.lib().dmrg_test_syevt(ctx.h, 1, (C.c_int * 1)(n), (C.c_int * 1)(n),
                                       A.ctypes.data_as(DP), w.ctypes.data_as(DP),
                                       U.ctypes.data_as(DP))
    assert code == 0, dmrgb.lib().dmrg_last_error(ctx.h)
    return w, U


@pytest.mark.parametrize("n,norm", [(n, s) for n in (41, 64, 100, 345, 600)
                                    for s in (1e-20, 1e-26, 1e-28, 1e-32, 1e-60, 1e-100, 1e30)]
                         + [(n, s) for n in (8, 24, 40) for s in (1e-26, 1e-32)])
def test_blocks_of_small_norm(dmrgb, ctx, n, norm):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    M = (Q * rng.uniform(0.05, 1.0, n)) @ Q.T
    M = 0.5 * (M + M.T)
    w, U = _values(dmrgb, ctx, M * norm)
    w = w / norm
    top = np.linalg.norm(M, 2)
    assert np.max(np.abs(w - np.linalg.eigvalsh(M)[::-1])) <= 2e-14 * max(1, n / 512) * top
    assert np.max(np.abs(U.T @ U - np.eye(n))) <= 1e-13
    assert np.max(np.abs(M @ U - U * w)) <= 1e-12 * top


@pytest.mark.parametrize("scale", [1e-40, 1e-26, 1e26, 1e60])
@pytest.mark.parametrize("krylov", [3, 8, 16])
def test_energy_scales_with_the_operator(dmrgb, ctx, krylov, scale):
    """The ground state of scale * H from the same start, betatest far below its Krylov elements:
    the energy is scale times that of H, to the 1e-9 that two sweeps leave of a converged energy."""
    L = 8
    base = dmrgb.makeMPO(dmrgb.heisenbergMPO, 2, L)
    e = []
    for f in (1.0, scale):
        mpo = dmrgb.makeMPO(dmrgb.heisenbergMPO, 2, L)
        mpo.W[0] = base.W[0] * f
        psi = dmrgb.randMPS(2, L, 16, seed=5)
        dev = dmrgb.DeviceState(psi, mpo.device(ctx))
        dev.env_build()
        p = dmrgb.make_params(maxm=16, krylov=krylov, betatest=1e-10 * f)
        e.append([dev.sweep(p) for _ in range(4)][-1]["energy"] / f)
    assert abs(e[1] - e[0]) <= 1e-9 * abs(e[0])
