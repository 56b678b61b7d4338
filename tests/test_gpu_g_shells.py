"""Shells up to g: classes whose working set is larger than a block's shared
memory, against the C++ restatement.

The transfers of a g shell expand fourth powers of the centres' separation (up
to 2 bohr: 16), so the f-shell bound of 1e-12 becomes 1e-11; in FP32 some tens
of roundings of 6e-8 times 16 stay below 1e-4 of the largest element (classes
with a g shell stay FP64 in a mixed build: in FP32 they do not).
"""
import numpy as np
import pytest

from origo_tlno_b200 import _native as N
from origo_tlno_b200 import engine as E
from origo_tlno_b200 import molecules as M
from oracle import port

pytestmark = pytest.mark.gpu


def _molecule():
    xyz = np.array([[0.0, 0.0, 0.0], [0.9, -0.5, 1.4]])
    mol = M.Molecule("g", np.array([6, 8]), xyz)
    for atom, L, exps in ((0, 0, [1.3]), (0, 4, [0.7, 2.1]), (1, 2, [0.8]), (1, 3, [1.1]), (1, 4, [0.9])):
        mol.shells.append(M.ShellSpec(tuple(xyz[atom]), L, np.array(exps), np.full(len(exps), 0.6), atom))
    return mol


@pytest.fixture(scope="module")
def case():
    if not port.available():
        pytest.skip("oracle not built")
    mol = _molecule()
    basis = port.PortBasis(mol)
    D = M.random_density(mol.n_sph, mol.n_sph // 3, seed=2)
    return mol, D, basis, basis.jk(D, tau=0.0)


def _close(out, ref, tol):
    return all(np.max(np.abs(out[k] - ref[k])) < tol for k in ("J", "K"))


def test_jk_with_g_shells(case):
    mol, D, basis, ref = case
    ctx = E.Context(mol).plan(E.ScreeningOptions(integral_threshold=0.0, mixed_threshold=1e6))
    assert np.max(np.abs(ctx.schwarz() - basis.schwarz())) < 1e-11
    assert _close(ctx.jk(D), ref, 1e-11)
    assert _close(ctx.jk(D, mixed=True), ref, 1e-4 * max(np.max(np.abs(ref[k])) for k in ("J", "K")))
    ctx.close()


def test_warp_forms_take_global_scratch(case):
    # without projector tables, or with a warp form asked for, also captured
    import torch
    mol, D, _, ref = case
    ctx = E.Context(mol)
    d = torch.tensor(D, device="cuda")
    J, K = torch.empty_like(d), torch.empty_like(d)
    for limit, warps in ((0, 0), (1 << 34, 1), (1 << 34, 8)):
        ctx.set_projector_limit(limit)
        ctx.set_tuning(generic_warps=warps)
        ctx.plan(E.ScreeningOptions(integral_threshold=0.0))
        assert _close(ctx.jk(D), ref, 1e-11)
        torch.cuda.synchronize()
        ctx.graph_capture(d.data_ptr(), J.data_ptr(), K.data_ptr())
        for _ in range(2):
            ctx.graph_launch()
        ctx.synchronize()
        assert _close({"J": J.cpu().numpy(), "K": K.cpu().numpy()}, ref, 1e-11)
    ctx.close()


def test_blocks_and_one_electron_matrices_with_g_shells(case):
    import torch
    mol, _, basis, _ = case
    ctx = E.Context(mol)
    quartets = [(1, 1, 1, 1), (1, 4, 4, 1), (4, 4, 4, 4), (4, 3, 1, 3), (1, 0, 4, 2), (2, 1, 3, 4)]
    for q, blk in zip(quartets, ctx.eri_blocks(quartets)):
        assert np.max(np.abs(blk - basis.eri_block(*q).reshape(blk.shape))) < 1e-11
    for a, b in zip(ctx.onee(), basis.onee()):
        assert np.max(np.abs(a - b)) < 1e-11
    # the allocation-free entry point has no room for such a quartet and says so
    q, off = np.array([[1, 1, 1, 1]], dtype=np.int32), np.zeros(1, dtype=np.int64)
    out = torch.empty(9 ** 4, device="cuda", dtype=torch.float64)
    with pytest.raises(E.TlnoError, match="eri_blocks_noalloc"):
        N.check(N.lib().tlno_gpu_eri_blocks_noalloc(ctx.h, 1, N.ptr(q), N.ptr(off), out.data_ptr()))
    ctx.close()
