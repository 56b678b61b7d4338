"""Rys roots as the compile-time kernels evaluate them."""
import numpy as np
import pytest

from origo_tlno_b200 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["fp64_fast", "fp32_fast"])
@pytest.mark.parametrize("n", range(1, 6))
def test_nan_argument_gives_nan(path, n):
    # the product of two exponents may overflow FP32, and at zero distance the
    # argument is then NaN: no table is indexed with its bits
    T = np.full(33, np.nan)
    T[::2] = 1.5
    r, w = E.rys_roots(T, n, path=path)
    assert np.all(np.isnan(r[1::2])) and np.all(np.isnan(w[1::2]))
    assert np.all(np.isfinite(r[::2])) and np.all(np.isfinite(w[::2]))
