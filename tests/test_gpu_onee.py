"""One-electron matrices on a kept context."""
import numpy as np
import pytest

from origo_tlno_b200 import engine as E
from origo_tlno_b200 import molecules as M

pytestmark = pytest.mark.gpu


def test_other_thresholds_on_a_kept_context():
    # the pair list is kept while the thresholds stay; a context evaluated at
    # one pair after another gives what a new context gives at each
    mol = M.cfg1()
    kept = E.Context(mol)
    loose = 0
    for decay, nuclear in [(1e-15, 1e-15), (1e-4, 1e-15), (1e-4, 1e-15), (1e-4, 1e-3), (1e-15, 1e-3),
                           (0.0, 0.0), (1e-15, 1e-15)]:
        kept.set_onee_thresholds(decay, nuclear)
        new = E.Context(mol)
        new.set_onee_thresholds(decay, nuclear)
        for screening in (True, False, True):
            a, b = kept.onee(screening), new.onee(screening)
            assert all(np.array_equal(x, y) for x, y in zip(a, b)), (decay, nuclear, screening)
        full = new.onee(screening=False)
        loose += any(not np.array_equal(x, y) for x, y in zip(b, full))
        new.close()
    assert loose >= 3  # the thresholds of this list do change the matrices
    kept.close()
