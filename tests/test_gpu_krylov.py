"""The one-launch Krylov vector kernels against the general ones: vectors on either side of the
one-launch limit give energies that agree with the oracle, and the Krylov dimensions whose Ritz
rotations pair differently (odd, even, the largest) reach the same ground state. Tolerance: a
converged energy is second order in the state's error, so 1e-11 relative bounds rounding alone."""
import numpy as np
import pytest

from oracle import dmrg as od, ed, models as om

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("krylov", [3, 4, 5, 8, 16])
def test_krylov_dimensions_reach_the_ground_state(dmrgb, ctx, krylov):
    L = 10
    mpo = dmrgb.makeMPO(dmrgb.heisenbergMPO, 2, L)
    psi = dmrgb.randMPS(2, L, 16, seed=krylov)
    E = dmrgb.dmrg(psi, mpo, m=32, sweeps=8, cutoff=0.0, krylov=krylov, ctx=ctx)
    E0 = ed.sparse_ground_energy(om.make_mpo([om.heisenberg_bulk()] * L, 2))
    assert abs(E - E0) <= 1e-11 * abs(E0)


@pytest.mark.parametrize("m", [45, 64, 91, 128, 129])
@pytest.mark.parametrize("krylov", [2, 6])
def test_vectors_around_the_one_launch_limits(dmrgb, ctx, m, krylov):
    """Two-site vectors of 4 m^2 elements: one, two, four and eight rounds over the cluster
    (m = 45, 64, 91, 128) and the general kernels (m = 129), one sweep against the oracle."""
    L = 16
    mpo = dmrgb.makeMPO(dmrgb.heisenbergMPO, 2, L)
    psi = dmrgb.randMPS(2, L, m, seed=m)
    ref = [np.array(a) for a in psi.tensors]
    E = dmrgb.dmrg(psi, mpo, m=m, sweeps=1, cutoff=1e-8, krylov=krylov, ctx=ctx)
    E0, info = od.dmrg(ref, om.make_mpo([om.heisenberg_bulk()] * L, 2), m=m, sweeps=1,
                       cutoff=1e-8, krylov=krylov, trunc="rho")
    assert abs(E - E0) <= 1e-9 * abs(E0)
    assert abs(psi.sweep_stats[-1]["entropy"] - info["sweeps"][-1]["entropy"]) <= 1e-8
