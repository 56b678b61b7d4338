"""The FP32 pass on small split schedules against the C++ restatement.

A split threshold far above every quartet's bound sends all of them to the FP32
kernels: lanes sharing a quartet, asynchronous density slots, J[ab] through
shared memory, the row kernel (f shells).  An FP32 integral carries some tens of
roundings of 6e-8 relative to its largest intermediate, which cancellation in
the transfers makes up to ten times the value, and J and K sum up to a few
hundred of them: 1e-5 of the largest element bounds that, and anything wrong in
a slot, a shuffle or an index is of the order of the elements.
"""
import numpy as np
import pytest

from origo_tlno_b200 import engine as E
from origo_tlno_b200 import molecules as M
from oracle import port
from tests.test_gpu_tiles import _molecule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [
    [(0, 1), (1, 1)], [(0, 2), (1, 3)], [(0, 5), (1, 1), (2, 2)], [(0, 9), (1, 2), (2, 1)],
    [(0, 12), (1, 5)], [(0, 1), (1, 5), (2, 2)], [(0, 3), (2, 2), (3, 1)],
    [(1, 2), (2, 1), (3, 2)],
], ids=lambda c: "-".join(f"{'spdf'[l]}{n}" for l, n in c))
def test_fp32_pass_matches_oracle(counts):
    if not port.available():
        pytest.skip("oracle not built")
    mol = _molecule(counts, seed=len(counts) + 10 * counts[0][1])
    D = M.random_density(mol.n_sph, max(1, mol.n_sph // 2), seed=9)
    ref = port.PortBasis(mol).jk(D)
    ctx = E.Context(mol).plan(E.ScreeningOptions(integral_threshold=0.0, mixed_threshold=1e6))
    assert np.max(ctx.schwarz()) ** 2 < 1e6 / np.max(np.abs(D))  # every quartet is below the split
    out, mixed = ctx.jk(D), ctx.jk(D, mixed=True)
    ctx.close()
    for key in ("J", "K"):
        top = float(np.max(np.abs(ref[key])))
        err = float(np.max(np.abs(out[key] - ref[key]))) / top
        err32 = float(np.max(np.abs(mixed[key] - ref[key]))) / top
        print(f"PIN fp32_pass {key}={err32:.2e} fp64={err:.2e}")
        assert 100 * err < err32 < 1e-5  # FP32 did run, and right
