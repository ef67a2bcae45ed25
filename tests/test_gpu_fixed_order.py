"""Solves whose sums keep one order give the numbers on record (tests/golden/fixed_order.json),
sweep for sweep. The 32-bit products of a split-precision solve turn any other last bit of a kept
vector into a difference of about 1e-8, which unconverged sweeps multiply, and sweeps of eight
Krylov vectors on long chains multiply last bits alike, so the order of every sum on their path is
part of their results. The starts are product states, which have no rounding of their own. The
record and the solve are the same arithmetic, so they agree to the rounding of the entropy's
logarithm, 1e-13; a rotation of nearly equal kept vectors shows at 1e-11 and above.
``python tests/test_gpu_fixed_order.py`` prints the record of the present engine."""
import json
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).resolve().parent / "golden" / "fixed_order.json"

# the largest density-matrix blocks have 84 to 170 states (U(1)) and 128 to 360 (dense), on either
# side of the line between the two kernels of one CTA per block
RAMPS = {"u1": [40, 90, 150], "tfi": [24, 64, 180]}
CASES = [dict(model=model, L=L, krylov=k, precision=prec) for model in RAMPS
         for L, k in ((20, 2), (26, 2), (20, 8)) for prec in ("3xtf32", "bf16x9")]
CASES += [dict(model=model, L=48, krylov=8, precision="fp64") for model in RAMPS]


def solve(pkg, ctx, model, L, krylov, precision):
    if model == "u1":
        mpo = pkg.makeMPO(pkg.heisenbergMPO, 2, L).with_qn(pkg.SPIN_QN)
        psi = pkg.neelMPS(L)
    else:
        mpo = pkg.makeMPO(pkg.tfiMPO(h=0.9), 2, L)
        psi = pkg.MPS([np.full((1, 2, 1), 2.0 ** -0.5) for _ in range(L)], oc=0)
    for i in range(L):                   # a field along z without symmetry
        mpo.W[i][-1, :, :, 0] += 0.125 * ((i * 7) % 5 - 2) * np.diag([0.5, -0.5])
    pkg.dmrg(psi, mpo, m=RAMPS[model], cutoff=1e-13, krylov=krylov, precision=precision, ctx=ctx)
    return [[s["energy"], s["max_truncerr"], s["entropy"], *map(float, s["d_top"])]
            for s in psi.sweep_stats]


def name(case):
    return f"{case['model']}-{case['L']}-{case['krylov']}-{case['precision']}"


@pytest.mark.parametrize("case", CASES, ids=name)
def test_sweeps_repeat_the_record(dmrgb, ctx, case):
    want = np.array(json.loads(GOLDEN.read_text())[name(case)])
    got = np.array(solve(dmrgb, ctx, **case))
    assert got.shape == want.shape
    assert np.max(np.abs(got - want) / np.maximum(np.abs(want), 1e-3)) <= 1e-13


if __name__ == "__main__":
    sys.path.insert(0, str(Path(__file__).resolve().parent))
    from conftest import load_package
    package = load_package()
    json.dump({name(c): solve(package, package.Context(0), **c) for c in CASES}, sys.stdout, indent=1)
