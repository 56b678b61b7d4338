"""Tile shapes of the ERI kernels against the C++ restatement.

Small molecules make the schedule share a quartet's primitive loops between
lanes and shorten the bra blocks; the primitive counts cover one, remainders
of every lane count, and more bra than ket primitives; two f shells of two
primitives pass one item batch of the block-per-quartet kernel.  FP64 sums of at most
a few thousand terms of magnitude <= 10 are exact to 1e-12.
"""
import numpy as np
import pytest

from origo_tlno_b200 import engine as E
from origo_tlno_b200 import molecules as M
from oracle import port

pytestmark = pytest.mark.gpu


def _molecule(counts, seed):
    rng = np.random.default_rng(seed)
    xyz = np.array([[0.0, 0.0, 0.0], [1.1, -0.4, 1.7]])
    mol = M.Molecule("tiles", np.array([6, 8]), xyz)
    for a in range(2):
        for L, n in counts:
            e = np.exp(rng.uniform(np.log(0.2), np.log(20.0), size=n))
            mol.shells.append(M.ShellSpec(tuple(xyz[a]), L, e, rng.uniform(0.1, 1.0, size=n), a))
    return mol


@pytest.mark.parametrize("counts", [
    [(0, 1), (1, 1)], [(0, 2), (1, 3)], [(0, 5), (1, 1), (2, 2)], [(0, 9), (1, 2), (2, 1)],
    [(0, 12), (1, 5)], [(0, 1), (1, 5), (2, 2)], [(0, 3), (2, 2), (3, 1)],
    [(1, 2), (2, 1), (3, 2)],
], ids=lambda c: "-".join(f"{'spdf'[l]}{n}" for l, n in c))
def test_split_tiles_match_oracle(counts):
    if not port.available():
        pytest.skip("oracle not built")
    mol = _molecule(counts, seed=len(counts) + 10 * counts[0][1])
    D = M.random_density(mol.n_sph, max(1, mol.n_sph // 2), seed=9)
    ref = port.PortBasis(mol).jk(D)
    ctx = E.Context(mol).plan(E.ScreeningOptions(integral_threshold=0.0))
    out = ctx.jk(D)
    mixed = ctx.jk(D, mixed=True)
    ctx.close()
    for key in ("J", "K"):
        err = float(np.max(np.abs(out[key] - ref[key])))
        err32 = float(np.max(np.abs(mixed[key] - ref[key])))
        print(f"PIN split_tiles {key}={err:.2e} mixed={err32:.2e}")
        assert err < 1e-12 and err32 < 1e-7
