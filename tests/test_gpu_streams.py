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


@pytest.mark.parametrize("mixed", [False, True])
def test_stream_counts_match_one_stream(mixed):
    # launches in order on one stream, over 4 and over the plan's own number (8);
    # context, captured graph and batch
    import torch
    mol = M.cfg1()
    D = M.density_for("cfg1", mol)
    d = torch.tensor(D, device="cuda")
    ctx = E.Context(mol).plan(E.ScreeningOptions(integral_threshold=1e-12, mixed_threshold=1e-7))
    # a batch short enough for the automatic rule to spread it
    ctxs = [E.Context(M.water_cluster(n, seed=5, grid=(2, 2, 2))) for n in (1, 3, 2)]
    b = E.Batch(ctxs, E.ScreeningOptions(integral_threshold=1e-12, mixed_threshold=1e-7))
    dens = [M.random_density(c.M, max(1, c.M // 4), seed=70 + i) for i, c in enumerate(ctxs)]
    out = {}
    for streams in (1, 4, 0):
        ctx.set_tuning(streams=streams)
        b.set_tuning(streams=streams)
        assert ctx.build_streams(mixed) == b.build_streams(mixed) == (streams or 8)
        one = ctx.jk(D, mixed=mixed)
        J, K = torch.empty_like(d), torch.empty_like(d)
        torch.cuda.synchronize()
        ctx.graph_capture(d.data_ptr(), J.data_ptr(), K.data_ptr(), mixed=mixed)
        ctx.graph_launch()
        ctx.synchronize()
        Jb, Kb = b.jk(dens, mixed=mixed)
        out[streams] = [one["J"], one["K"], J.cpu().numpy(), K.cpu().numpy(), *Jb, *Kb]
    for streams in (4, 0):
        assert max(_maxabs(x, y) for x, y in zip(out[streams], out[1])) < 1e-12
    b.close()
    ctx.close()


def test_threads_build_beside_each_other():
    # every host thread has auxiliary streams of its own: two threads build and
    # replay on their own contexts at once and get what each gets alone
    import threading
    import torch
    work = []
    for k, mol in enumerate((M.cfg1(), M.water_cluster(4, seed=5, grid=(2, 2, 2)))):
        D = M.random_density(mol.n_sph, max(1, mol.n_sph // 5), seed=40 + k)
        ctx = E.Context(mol).plan(E.ScreeningOptions(integral_threshold=1e-12))
        ctx.set_tuning(streams=1)
        ref = ctx.jk(D)
        ctx.set_tuning()
        assert ctx.build_streams() == 8
        d = torch.tensor(D, device="cuda")
        work.append((ctx, D, ref, d, torch.empty_like(d), torch.empty_like(d)))
    torch.cuda.synchronize()
    worst, failed = [0.0, 0.0], []
    start = threading.Barrier(2)

    def build(i):
        try:
            ctx, D, ref, d, J, K = work[i]
            start.wait(60)
            for _ in range(40):
                out = ctx.jk(D)
                ctx.graph_capture(d.data_ptr(), J.data_ptr(), K.data_ptr())
                ctx.graph_launch()
                ctx.synchronize()
                worst[i] = max(worst[i], _maxabs(out["J"], ref["J"]), _maxabs(out["K"], ref["K"]),
                               _maxabs(J.cpu().numpy(), ref["J"]), _maxabs(K.cpu().numpy(), ref["K"]))
        except Exception as e:  # reported below, in the test's own thread
            failed.append(e)

    threads = [threading.Thread(target=build, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    assert max(worst) < 1e-12
    # a captured graph outlives the thread, and its streams, that captured it
    for ctx, D, ref, d, J, K in work:
        J.zero_(), K.zero_()
        torch.cuda.synchronize()
        ctx.graph_launch()
        ctx.synchronize()
        assert max(_maxabs(J.cpu().numpy(), ref["J"]), _maxabs(K.cpu().numpy(), ref["K"])) < 1e-12
        ctx.close()
