"""Builds whose class launches run on several streams."""
import numpy as np
import pytest

from origo_tlno_b200 import engine as E
from origo_tlno_b200 import molecules as M

pytestmark = pytest.mark.gpu


def _maxabs(a, b):
    return float(np.max(np.abs(a - b)))


def test_failed_build_leaves_nothing_running_beside_its_stream():
    # a build that fails between its class launches has already queued some on
    # auxiliary streams; waiting for the context's stream covers them, so J and
    # K no longer change, and the next build and capture are whole
    import torch
    mol = M.cfg1()
    D = M.density_for("cfg1", mol)
    ctx = E.Context(mol).plan(E.ScreeningOptions(integral_threshold=1e-12))
    ref = ctx.jk(D)
    n = len(ctx.combos())
    d = torch.tensor(D, device="cuda")
    J, K = torch.zeros_like(d), torch.zeros_like(d)
    torch.cuda.synchronize()
    for after in (1, n // 2, n - 1):
        ctx.fail_next_build(after)
        with pytest.raises(E.TlnoError, match="injected"):
            ctx.jk_device(d.data_ptr(), J.data_ptr(), K.data_ptr())
        ctx.synchronize()
        seen = J.clone(), K.clone()
        torch.cuda.synchronize()
        assert torch.equal(seen[0], J) and torch.equal(seen[1], K)
        ctx.fail_next_build(after)
        with pytest.raises(E.TlnoError, match="injected"):
            ctx.graph_capture(d.data_ptr(), J.data_ptr(), K.data_ptr())
    ctx.jk_device(d.data_ptr(), J.data_ptr(), K.data_ptr())
    assert max(_maxabs(J.cpu().numpy(), ref["J"]), _maxabs(K.cpu().numpy(), ref["K"])) < 1e-12
    J.zero_(), K.zero_()
    torch.cuda.synchronize()
    ctx.graph_capture(d.data_ptr(), J.data_ptr(), K.data_ptr())
    ctx.graph_launch()
    ctx.synchronize()
    assert max(_maxabs(J.cpu().numpy(), ref["J"]), _maxabs(K.cpu().numpy(), ref["K"])) < 1e-12
    ctx.close()
