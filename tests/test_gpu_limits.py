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
