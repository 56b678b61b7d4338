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


def test_tuning_another_knob_keeps_the_streams_of_the_plans_size():
    # streams 0 (the default) means by the plan's size: it can be set back, and
    # setting another knob does not put a short build on one stream
    ctx = E.Context(M.cfg1()).plan(E.ScreeningOptions(integral_threshold=1e-12))
    auto = ctx.build_streams()
    assert auto == 8 and ctx.build_streams(mixed=True) == 8
    ctx.set_tuning(grid_mult=8)
    assert ctx.build_streams() == auto
    for n in (1, 4):
        ctx.set_tuning(streams=n)
        assert ctx.build_streams() == n
    ctx.set_tuning(streams=0)
    assert ctx.build_streams() == auto
    b = E.Batch([ctx], E.ScreeningOptions(integral_threshold=1e-12))
    b.set_tuning(streams=2)
    assert b.build_streams() == 2
    b.set_tuning()
    assert b.build_streams() == auto
    for bad in (-1, 5):
        with pytest.raises(E.TlnoError, match="out of range"):
            ctx.set_tuning(streams=bad)
        with pytest.raises(E.TlnoError, match="out of range"):
            b.set_tuning(streams=bad)
    b.close()
    ctx.close()
