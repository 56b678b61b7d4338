"""Limits and refusals of the J/K plans."""
import numpy as np
import pytest

from origo_tlno_b200 import engine as E
from origo_tlno_b200 import molecules as M

pytestmark = pytest.mark.gpu


def test_batch_refuses_more_functions_than_the_matrix_indices_hold():
    # the kernels index a matrix with 32 bits (M <= 65535): a batch refuses a
    # larger molecule as a single context does, before any pair is formed
    n = 9363  # f shells: 65541 functions
    mol = M.Molecule("large", np.array([1]), np.zeros((1, 3)))
    mol.shells = [M.ShellSpec((0.0, 0.0, 0.01 * k), 3, np.array([1.0]), np.array([1.0]), 0) for k in range(n)]
    big, small = E.Context(mol), E.Context(M.cfg0())
    assert big.M == 7 * n > 65535
    with pytest.raises(E.TlnoError, match="M <= 65535"):
        big.plan()
    with pytest.raises(E.TlnoError, match="M <= 65535"):
        E.Batch([small, big])
    big.close()
    small.close()


def test_projector_limit_and_warp_form_give_the_same_matrices():
    # with less memory than the projector tables need the largest go first; the
    # classes without one run warp per quartet, (dd|dp) and (fp|dp) then keep
    # their compile-time kernels, and a warp form asked for leaves the classes
    # the block kernel took over from a compile-time one where they are
    mol = M.fragment(M.cfg2(), [0, 1, 2])
    D = M.random_density(mol.n_sph, max(1, mol.n_sph // 5), seed=3)
    opts = E.ScreeningOptions(integral_threshold=1e-12)
    ctx = E.Context(mol).plan(opts)
    ref, mixed = ctx.jk(D), ctx.jk(D, mixed=True)
    n_fast = sum(c["fast"] for c in ctx.combos())
    for limit in (0, 20000, 400000, 4000000, 1 << 34):
        ctx.set_projector_limit(limit)
        ctx.plan(opts)
        assert sum(c["fast"] for c in ctx.combos()) >= n_fast
        out, out32 = ctx.jk(D), ctx.jk(D, mixed=True)
        for k in ("J", "K"):
            assert np.max(np.abs(out[k] - ref[k])) < 1e-12
            assert np.max(np.abs(out32[k] - mixed[k])) < 1e-7
    for warps in (1, 4):
        ctx.set_tuning(generic_warps=warps)
        for replan in (False, True):
            if replan:
                ctx.plan(opts)
            out = ctx.jk(D)
            assert max(np.max(np.abs(out[k] - ref[k])) for k in ("J", "K")) < 1e-12
    with pytest.raises(E.TlnoError, match="limit"):
        ctx.set_projector_limit(-1)
    ctx.close()


def test_batch_of_one_molecule_matches_its_context():
    import torch
    mol = M.water_cluster(2, seed=5, grid=(2, 1, 1))
    D = M.random_density(mol.n_sph, max(1, mol.n_sph // 5), seed=6)
    for opts in (E.ScreeningOptions(integral_threshold=1e-12, mixed_threshold=1e-6),
                 E.ScreeningOptions(integral_threshold=1e-12, density_threshold=1e-9)):
        ctx = E.Context(mol).plan(opts)
        b = E.Batch([ctx], opts)
        for mixed in (False, True):
            ref = ctx.jk(D, mixed=mixed)
            J, K = b.jk([D], mixed=mixed)
            assert max(np.max(np.abs(J[0] - ref["J"])), np.max(np.abs(K[0] - ref["K"]))) < 1e-12
            d = torch.tensor(D, device="cuda")
            dJ, dK = torch.empty_like(d), torch.empty_like(d)
            torch.cuda.synchronize()
            b.graph_capture(d.data_ptr(), dJ.data_ptr(), dK.data_ptr(), mixed=mixed)
            b.graph_launch()
            b.synchronize()
            assert max(np.max(np.abs(dJ.cpu().numpy() - ref["J"])), np.max(np.abs(dK.cpu().numpy() - ref["K"]))) < 1e-12
        b.close()
        ctx.close()


def test_plan_of_a_contraction_beyond_31_bits():
    # one shell of 220 primitives: 48400 primitive pairs, 2.3e9 primitive
    # quartets in its one tile (planned with the decay metric, which evaluates
    # no integral; the build itself is not run)
    mol = M.Molecule("deep", np.array([1]), np.zeros((1, 3)))
    mol.shells = [M.ShellSpec((0.0, 0.0, 0.0), 0, np.geomspace(0.1, 1e4, 220), np.ones(220), 0)]
    ctx = E.Context(mol).plan(E.ScreeningOptions(integral_threshold=0.0, decay_threshold=1e-10))
    assert ctx.profile()["primitive_quartets"] == 48400 ** 2
    ctx.close()
