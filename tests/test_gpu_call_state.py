"""What one call leaves behind for the next: counters, error records, marked slots."""
import numpy as np
import pytest

from skywalker_b200 import APP_PPR, MODE_ONLINE, WALK_UNBIASED
from skywalker_b200.api import SkwError

pytestmark = pytest.mark.gpu


def _device_batch(starts, hop):
    import torch
    n = len(starts)
    return (torch.from_numpy(starts.view(np.int32)).cuda(), torch.zeros(n * hop, dtype=torch.int32, device="cuda"),
            torch.zeros(n, dtype=torch.int32, device="cuda"))


@pytest.mark.parametrize("before", ["upload", "save"])
@pytest.mark.parametrize("kw", [dict(flags=WALK_UNBIASED), dict(mode=MODE_ONLINE)])
def test_queued_walks_leave_no_edges_to_the_next_call(ctx, oracle, rmat12, tmp_path, before, kw):
    """The resident graph's largest degree and a checkpoint's fingerprint pass through the word in which synchronous
    calls count their edges; queued walks in between must not make the next call find them there."""
    g = rmat12
    starts = oracle.gen_starts(2000, g.V, 3)
    d_s, d_p, d_l = _device_batch(starts, 31)
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    if before == "save":
        ctx.alias_build_offline()
        ctx.alias_save(str(tmp_path / "t.skw"))
    ctx.walk(d_s, 31, app=APP_PPR, tp=0.1, seed=5, paths=d_p, lengths=d_l, enqueue_only=True, **kw)
    queued = ctx.take_sampled_edges()
    _, lens, _, edges = ctx.walk(starts, 31, app=APP_PPR, tp=0.1, seed=5, **kw)
    assert edges == int(lens.sum()) == queued
    _, sl, _, edges = ctx.sample_khop(starts[:100], [5, 3], mode=MODE_ONLINE)
    assert edges == int(sl.sum())


def _slots(ctx):
    """prob and alias of every slot as they are on the device."""
    import torch
    s = torch.as_tensor(ctx.alias_device_arrays()[0], device="cuda").cpu().numpy().view(np.uint32).reshape(-1, 2)
    return s[:, 0].copy().view(np.float32), s[:, 1].copy()


@pytest.mark.parametrize("first", ["truncated", "refused"])
def test_partial_build_after_a_table_that_failed(ctx, oracle, rmat12, tmp_path, first):
    """A checkpoint that ends too soon or an import that is refused leaves no slots that a build of a range would let
    pass as built: outside the range they say "no table"."""
    g = rmat12
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    path = str(tmp_path / "t.skw")
    ctx.alias_save(path)
    prob, alias, valid = ctx.alias_export()
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)          # new slots, in memory that held the table before
    with pytest.raises(SkwError):
        if first == "truncated":
            with open(path, "r+b") as f:
                f.truncate(48 + 8 * 100)
            ctx.alias_load(path)
        else:
            alias[-1] = 1 << 30
            ctx.alias_import(prob, alias, valid)
    half = g.V // 2
    ctx.alias_build_offline(0, half)
    got, _ = _slots(ctx)
    want, _, want_valid = oracle.alias_build(g.xadj, g.adjwgt)
    cut = int(g.xadj[half])
    assert (got[cut:] == -1.0).all()
    deg = np.diff(g.xadj.astype(np.int64))
    usable = np.repeat(want_valid.astype(bool), deg)[:cut]
    assert np.array_equal(got[:cut][usable], want[:cut][usable])
    assert not ctx.alias_export()[2][half:].any()


def test_partial_build_after_online_sampling(ctx, oracle, rmat12):
    """Online sampling leaves tables of the vertices it met; a build of a range starts from "no table" everywhere, in
    the flags as in the slots."""
    g = rmat12
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.sample_khop(oracle.gen_starts(500, g.V, 3), [5, 3], mode=MODE_ONLINE)
    half = g.V // 2
    ctx.alias_build_offline(0, half)
    prob, alias, valid = ctx.alias_export()
    want_prob, want_alias, want_valid = oracle.alias_build(g.xadj, g.adjwgt)
    assert np.array_equal(valid[:half], want_valid[:half])
    usable = np.repeat(valid.astype(bool), np.diff(g.xadj.astype(np.int64)))
    assert np.array_equal(prob[usable], want_prob[usable]) and np.array_equal(alias[usable], want_alias[usable])


@pytest.mark.parametrize("kw", [dict(), dict(mode=MODE_ONLINE), dict(mode=MODE_ONLINE, flags=4)])
def test_error_of_a_queued_walk_waits_for_its_own_report(ctx, oracle, rmat12, kw):
    """A synchronous call neither reports nor loses what a queued walk before it did wrong."""
    g = rmat12
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    starts = oracle.gen_starts(300, g.V, 3)
    want, want_len, _, want_edges = ctx.walk(starts, 11, seed=5)
    bad = starts.copy()
    bad[7] = g.V + 7
    d_s, d_p, d_l = _device_batch(bad, 11)
    ctx.walk(d_s, 11, seed=5, paths=d_p, lengths=d_l, enqueue_only=True, **kw)
    paths, lens, _, edges = ctx.walk(starts, 11, seed=5, **kw)
    assert np.array_equal(paths, want) and np.array_equal(lens, want_len) and edges == want_edges
    with pytest.raises(SkwError) as e:
        ctx.take_sampled_edges()
    assert "index out of range" in str(e.value)
    with pytest.raises(SkwError):                   # the synchronous call's own errors are its own
        ctx.walk(bad, 11, seed=5, **kw)
    ctx.walk(starts, 11, seed=5, **kw)
    assert ctx.take_sampled_edges() == 0


@pytest.mark.parametrize("kw", [dict(), dict(app=APP_PPR, tp=0.1), dict(flags=2)])
def test_rows_of_a_failed_walk_are_not_written(ctx, oracle, rmat12, kw):
    """A start vertex that does not exist fails the call; rows that are not to be filled keep what they held."""
    import torch
    g = rmat12
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    bad = oracle.gen_starts(300, g.V, 3)
    bad[7] = g.V + 7
    paths = torch.full((300, 11), 5, dtype=torch.int32).pin_memory()
    lengths = torch.zeros(300, dtype=torch.int32).pin_memory()
    with pytest.raises(SkwError):
        ctx.walk(bad, 11, seed=5, paths=paths, lengths=lengths, **kw)
    assert (paths == 5).all()


def test_class_counters_across_calls_and_streams(oracle, plaw):
    """Builds take zeroed counters from a few sets that the status kernel clears: more builds in one call than there are
    sets, queued builds whose call nothing waits for, and builds on another stream behind them."""
    import torch
    from skywalker_b200 import MODE_ONLINE
    from skywalker_b200.api import Context
    g = plaw
    c = Context(0)
    c.upload(g.xadj, g.adjncy, g.adjwgt)
    table = oracle.alias_build(g.xadj, g.adjwgt)
    n, hop = 20000, 21                              # 20 frontiers a call
    starts = oracle.gen_starts(n, g.V, 5)
    want, want_len = oracle.walk(g.xadj, g.adjncy, g.adjwgt, table, starts, hop, seed=8)
    s = torch.from_numpy(starts.view(np.int32)).cuda()
    p = torch.zeros((n, hop), dtype=torch.int32, device="cuda")
    l = torch.zeros(n, dtype=torch.int32, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    live = np.arange(hop)[None, :] <= want_len[:, None]

    def same():
        assert np.array_equal(l.cpu().numpy().view(np.uint32), want_len)
        assert np.array_equal(p.cpu().numpy().view(np.uint32)[live], want[live])

    for turn in range(4):
        c.set_stream(streams[turn % 2].cuda_stream)
        for flags in (0, 4, 0, 0):                  # tables of the whole graph, of every step's frontier
            c.walk(s, hop, seed=8, mode=MODE_ONLINE, paths=p, lengths=l, flags=flags, enqueue_only=True)
        c.set_stream(streams[1 - turn % 2].cuda_stream)
        c.alias_build_offline()
        prob, alias, valid = c.alias_export()
        assert np.array_equal(prob, table[0]) and np.array_equal(alias, table[1]) and np.array_equal(valid, table[2])
        torch.cuda.synchronize()
        same()
        for flags in (4, 0):
            p.zero_(), l.zero_()
            torch.cuda.synchronize()
            c.walk(s, hop, seed=8, mode=MODE_ONLINE, paths=p, lengths=l, flags=flags)
            same()
    c.close()
