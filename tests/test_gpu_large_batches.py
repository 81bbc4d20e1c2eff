"""Batches that are large enough for slices, host threads or tables of the whole graph."""
import numpy as np
import pytest

from skywalker_b200 import APP_DEEPWALK, APP_NODE2VEC, APP_PPR, MODE_OFFLINE, MODE_ONLINE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("app,kw", [(APP_DEEPWALK, {}), (APP_PPR, {"tp": 0.3}), (APP_NODE2VEC, {"p": 2.0, "q": 0.5})])
@pytest.mark.parametrize("n", [(1 << 18) + 3, (1 << 20) + 12345])      # one slice, two slices
def test_online_host_batches(ctx, oracle, plaw, app, kw, n):
    """Online walks with host results, packed and as rows, are the offline walks of the same seed."""
    g = plaw
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    starts = oracle.gen_starts(n, g.V, 5)
    want, want_len, want_cells, _, want_edges = ctx.walk_packed(starts, 6, app=app, seed=8, mode=MODE_OFFLINE, **kw)
    out, lens, cells, ms, edges = ctx.walk_packed(starts, 6, app=app, seed=8, mode=MODE_ONLINE, **kw)
    assert (cells, edges) == (want_cells, want_edges) and ms > 0
    assert np.array_equal(lens, want_len) and np.array_equal(out[:cells], want[:cells])
    rows, lens, _, edges = ctx.walk(starts, 6, app=app, seed=8, mode=MODE_ONLINE, **kw)
    live = np.arange(6)[None, :] <= lens[:, None]
    assert np.array_equal(lens, want_len) and edges == want_edges and np.array_equal(rows[live], want[:cells])
    table = oracle.alias_build(g.xadj, g.adjwgt)
    for w in range(0, n, n // 50):
        op, ol = oracle.walk(g.xadj, g.adjncy, g.adjwgt, table, starts[w:w + 1], 6, app=app, seed=8, walker_base=int(w), **kw)
        assert ol[0] == lens[w] and np.array_equal(op[0, :ol[0] + 1], rows[w, :ol[0] + 1])


@pytest.mark.parametrize("warm", [0, 300, 40000])      # walkers of the call before: none, slots computed, tables
def test_captured_online_walk(oracle, plaw, warm):
    """A queued online walk captured into a graph and replayed, before and after calls that take tables."""
    import torch
    from skywalker_b200.api import Context
    g = plaw
    n, hop = 40000, 21
    c = Context(0)
    c.upload(g.xadj, g.adjncy, g.adjwgt)
    starts = oracle.gen_starts(n, g.V, 5)
    table = oracle.alias_build(g.xadj, g.adjwgt)
    want, want_len = oracle.walk(g.xadj, g.adjncy, g.adjwgt, table, starts, hop, seed=8)
    live = np.arange(hop)[None, :] <= want_len[:, None]
    s = torch.from_numpy(starts.view(np.int32)).cuda()
    p = torch.zeros((n, hop), dtype=torch.int32, device="cuda")
    l = torch.zeros(n, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    c.set_stream(stream.cuda_stream)
    kw = dict(mode=MODE_ONLINE, seed=8, paths=p, lengths=l, enqueue_only=True)
    if warm:
        c.walk(s, hop, n=warm, **kw)
        c.take_sampled_edges()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        c.walk(s, hop, **kw)
    for _ in range(2):
        p.zero_(), l.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        assert c.take_sampled_edges() == int(want_len.sum())
        assert np.array_equal(l.cpu().numpy(), want_len)
        assert np.array_equal(p.cpu().numpy().view(np.uint32)[live], want[live])
        c.walk(starts, hop, mode=MODE_ONLINE, seed=9)
    del graph
    c.close()


@pytest.mark.parametrize("flags", [0, 4])
def test_queued_online_walks_on_two_streams(oracle, plaw, flags):
    """Queued walks that build tables, one behind the other on different streams, and a table built meanwhile."""
    import torch
    from skywalker_b200.api import Context
    g = plaw
    n, hop = 40000, 11
    c = Context(0)
    c.upload(g.xadj, g.adjncy, g.adjwgt)
    starts = oracle.gen_starts(n, g.V, 5)
    table = oracle.alias_build(g.xadj, g.adjwgt)
    streams = [torch.cuda.Stream() for _ in range(2)]
    s = torch.from_numpy(starts.view(np.int32)).cuda()
    outs = [(torch.zeros((n, hop), dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda"))
            for _ in range(6)]
    torch.cuda.synchronize()
    for i, (p, l) in enumerate(outs):
        c.set_stream(streams[i % 2].cuda_stream)
        c.walk(s, hop, mode=MODE_ONLINE, flags=flags, seed=i, paths=p, lengths=l, enqueue_only=True)
    c.set_stream(0)
    c.alias_build_offline()
    prob, alias, valid = c.alias_export()
    assert np.array_equal(valid, table[2]) and np.array_equal(prob, table[0]) and np.array_equal(alias, table[1])
    torch.cuda.synchronize()
    total = 0
    for i, (p, l) in enumerate(outs):
        want, want_len = oracle.walk(g.xadj, g.adjncy, g.adjwgt, table, starts, hop, seed=i)
        live = np.arange(hop)[None, :] <= want_len[:, None]
        assert np.array_equal(l.cpu().numpy(), want_len)
        assert np.array_equal(p.cpu().numpy().view(np.uint32)[live], want[live])
        total += int(want_len.sum())
    assert c.take_sampled_edges() == total
    c.close()


@pytest.mark.parametrize("app,kw", [(APP_DEEPWALK, {}), (APP_PPR, {"tp": 0.15})])
@pytest.mark.parametrize("n", [5000, (1 << 18) + 777])      # a copy of the matrix, host threads
def test_rows_made_by_the_library_are_filled(ctx, oracle, rmat12, app, kw, n):
    """Rows that the caller did not bring: cells past a walk's end hold INVALID_VERTEX, also in memory used before."""
    g = rmat12
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    starts = oracle.gen_starts(n, g.V, 31)
    table = oracle.alias_build(g.xadj, g.adjwgt)
    for seed in (8, 9):
        rows, lens, _, edges = ctx.walk(starts, 21, app=app, seed=seed, **kw)
        want, want_len = oracle.walk(g.xadj, g.adjncy, g.adjwgt, table, starts, 21, app=app, seed=seed, fill=0xFFFFFFFF, **kw)
        assert np.array_equal(lens, want_len) and edges == int(want_len.sum()) and np.array_equal(rows, want)
        rows[:] = 0x5A5A5A5A
        del rows, lens


@pytest.mark.parametrize("n", [1, 31, 63, 64, 65, 511, 512, 513])
def test_ppr_records_chunk_edges(ctx, oracle, rmat12, n):
    """The chunked kernel of PPR over records, which takes batches of more walkers than fit the GPU at a lane each: the
    walkers of the last chunk and CTA, paths that leave the staged cells, rows of several lines."""
    import torch
    g = rmat12
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    ctx.walk_records_build()
    table = oracle.alias_build(g.xadj, g.adjwgt)
    least = 700 * torch.cuda.get_device_properties(0).multi_processor_count
    n += (least + 511) // 512 * 512
    starts = oracle.gen_starts(n, g.V, n)
    paths, lens, _, edges = ctx.walk(starts, 40, app=APP_PPR, tp=0.02, seed=n, walker_base=7)
    want, want_len = oracle.walk(g.xadj, g.adjncy, g.adjwgt, table, starts, 40, app=APP_PPR, tp=0.02, seed=n, walker_base=7)
    live = np.arange(40)[None, :] <= want_len[:, None]
    assert np.array_equal(lens, want_len) and edges == int(want_len.sum()) and np.array_equal(paths[live], want[live])


@pytest.mark.parametrize("flags", [0, 2])
@pytest.mark.parametrize("n", [2516, 2517, 5032, 5033, 10064, 10065, 20129, 40257])
def test_deepwalk_walkers_a_warp_on_a_small_graph(ctx, oracle, rmat12, n, flags):
    """Batch sizes around which the number of walkers a warp changes on a graph whose tables are small."""
    g = rmat12
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    starts = oracle.gen_starts(n, g.V, 5)
    paths, lens, _, edges = ctx.walk(starts, 12, seed=8, flags=flags)
    table = oracle.alias_build(g.xadj, g.adjwgt) if flags == 0 else None
    want, want_len = oracle.walk(g.xadj, g.adjncy, g.adjwgt if flags == 0 else None, table, starts, 12, seed=8,
                                 **({} if flags == 0 else {"unbiased": True}))
    live = np.arange(12)[None, :] <= want_len[:, None]
    assert np.array_equal(lens, want_len) and edges == int(want_len.sum()) and np.array_equal(paths[live], want[live])


@pytest.mark.parametrize("graph", ["rmat16", "plaw"])                  # mostly dead ends, none
@pytest.mark.parametrize("hop,tp", [(1, 0.15), (2, 0.5), (8, 0.15), (9, 0.1), (10, 0.0), (81, 0.02), (101, 0.15)])
@pytest.mark.parametrize("n", [104001, (1 << 20) + 33])                # chunked PPR in one slice, in three
def test_packed_ppr_over_records(ctx, oracle, request, graph, hop, tp, n):
    """PPR over the records, packed: the first eight cells of the rows travel apart from the rest.  The same cells and
    lengths as the rows of the same call, at row lengths around eight, and as the oracle's walks."""
    import torch
    g = request.getfixturevalue(graph)
    if n > 1 << 20 and hop > 10:
        n = (1 << 20) // 8 * 8 + 1 if tp > 0.1 else 104001
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    ctx.walk_records_build()
    starts = oracle.gen_starts(n, g.V, 5)
    rows = torch.full((n, hop), -1, dtype=torch.int32, device="cuda")
    lens = torch.zeros(n, dtype=torch.int32, device="cuda")
    kw = dict(app=APP_PPR, tp=tp, seed=8, walker_base=3)
    s = torch.from_numpy(starts.view(np.int32)).cuda()
    torch.cuda.synchronize()
    _, _, _, edges = ctx.walk(s, hop, paths=rows, lengths=lens, **kw)
    rows, lens = rows.cpu().numpy().view(np.uint32), lens.cpu().numpy().view(np.uint32)
    live = np.arange(hop)[None, :] <= lens[:, None]
    want = rows[live]
    for u8 in (False, True):
        out, got, cells, ms, e = ctx.walk_packed(starts, hop, lengths_u8=u8, **kw)
        assert cells == len(want) and e == edges and ms > 0
        assert np.array_equal(got, lens) and np.array_equal(out[:cells], want)
    table = oracle.alias_build(g.xadj, g.adjwgt)
    op, ol = oracle.walk(g.xadj, g.adjncy, g.adjwgt, table, starts[:2000], hop, **kw)
    assert np.array_equal(ol, lens[:2000])
    keep = np.arange(hop)[None, :] <= ol[:, None]
    assert np.array_equal(op[keep], rows[:2000][keep])


@pytest.mark.parametrize("hop", [1, 2, 31, 32, 33, 81])
@pytest.mark.parametrize("app", [APP_DEEPWALK, APP_PPR])
@pytest.mark.parametrize("n,off,flags", [(1, 0, 0), (37, 5, 16), (4096, 31, 16), (4097, 2, 0), (9999, 1, 18)])
def test_rows_written_into_pinned_memory(ctx, oracle, rmat12, app, hop, n, off, flags):
    """Rows in the caller's pinned matrix, wherever in a 128-byte line a row starts (off words).  16, fill rows: DeepWalk and PPR write
    them there, a line at a time, and cells past a walk's end get the invalid vertex; otherwise the cells of the walks are
    copied, and those past their ends keep their contents.  Words around the matrix keep theirs, and all of it equals the rows of
    pageable memory; 2: uniform draws."""
    import torch
    g = rmat12
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    starts = oracle.gen_starts(n, g.V, 11)
    paths = torch.full((n * hop + 64,), 0x5A5A5A5A, dtype=torch.int32).pin_memory()
    lengths = torch.full((n + 2,), 0x5A5A5A5A, dtype=torch.int32).pin_memory()
    kw = dict(app=app, tp=0.1, seed=6, walker_base=9, flags=flags)
    _, _, ms, edges = ctx.walk(starts, hop, paths=paths[off:off + n * hop], lengths=lengths[1:n + 1], **kw)
    p, l = paths.numpy().view(np.uint32), lengths.numpy().view(np.uint32)
    rows, lens = p[off:off + n * hop].reshape(n, hop), l[1:n + 1]
    assert (p[:off] == 0x5A5A5A5A).all() and (p[off + n * hop:] == 0x5A5A5A5A).all()
    assert l[0] == l[-1] == 0x5A5A5A5A and ms > 0 and edges == int(lens.sum())
    live = np.arange(hop)[None, :] <= lens[:, None]
    assert (rows[~live] == (0xFFFFFFFF if flags & 16 else 0x5A5A5A5A)).all()
    wp, wl = np.zeros((n, hop), np.uint32), np.zeros(n, np.uint32)
    _, _, _, e = ctx.walk(starts, hop, paths=wp, lengths=wl, **kw)
    assert e == edges and np.array_equal(wl, lens) and np.array_equal(wp[live], rows[live])
    # not at a word boundary: pinned memory as well, but copied
    odd = torch.zeros(n * hop * 4 + 4, dtype=torch.uint8).pin_memory().numpy()[2:2 + n * hop * 4].view(np.uint32)
    ctx.walk(starts, hop, paths=odd, lengths=wl, **kw)
    assert np.array_equal(odd.reshape(n, hop)[live], rows[live])


@pytest.fixture(scope="module")
def rmat19(ctx):
    """Tables out of cache (72 MB), on the host as well."""
    ctx.generate_rmat(19, 12 << 19, graph_seed=2, weight_seed=3)
    x, a, w = ctx.download()
    assert len(a) * 12 > 64 << 20
    return x, a, w


@pytest.mark.parametrize("app,hop,n,off,flags", [
    (APP_DEEPWALK, 81, 4099, 7, 16), (APP_DEEPWALK, 81, 4099, 7, 0), (APP_DEEPWALK, 11, 2500, 31, 16), (APP_DEEPWALK, 70, 16281, 1, 16),
    (APP_PPR, 81, 4099, 5, 16), (APP_PPR, 33, 9999, 3, 16)])
def test_rows_written_into_pinned_memory_of_a_large_graph(ctx, oracle, rmat19, app, hop, n, off, flags):
    """The same where draws fetch their neighbours ahead, into an array that the caller has registered."""
    import mmap
    import torch
    x, a, w = rmat19
    ctx.upload(x, a, w)
    ctx.alias_build_offline()
    starts = oracle.gen_starts(n, len(x) - 1, 12)
    cells = np.frombuffer(mmap.mmap(-1, (n * hop + 64 + n) * 4), np.uint32)
    cells[:] = 0x5A5A5A5A
    rows, lengths = cells[off:off + n * hop].reshape(n, hop), cells[n * hop + 64:]
    kw = dict(app=app, tp=0.1, seed=6, walker_base=9)
    runtime = torch.cuda.cudart()
    assert int(runtime.cudaHostRegister(cells.ctypes.data, cells.nbytes, 0)) == 0
    try:
        ctx.walk(starts, hop, paths=rows, lengths=lengths, flags=flags, **kw)
    finally:
        runtime.cudaHostUnregister(cells.ctypes.data)
    want, want_len = oracle.walk(x, a, w, ctx.alias_export(), starts, hop, **kw)
    live = np.arange(hop)[None, :] <= want_len[:, None]
    assert np.array_equal(lengths, want_len) and np.array_equal(rows[live], want[live])
    assert (rows[~live] == (0xFFFFFFFF if flags else 0x5A5A5A5A)).all()
    assert (cells[:off] == 0x5A5A5A5A).all() and (cells[off + n * hop:n * hop + 64] == 0x5A5A5A5A).all()


@pytest.mark.parametrize("hop", [1, 2, 31, 32, 33, 40])
@pytest.mark.parametrize("app", [APP_DEEPWALK, APP_PPR])
@pytest.mark.parametrize("n,flags", [(4097, 18), (9999, 16)])
def test_short_rows_written_into_pinned_memory(ctx, oracle, rmat12, app, hop, n, flags):
    """Rows of a line or less with uniform draws (2), and those a little longer of draws from tables in cache."""
    import torch
    g = rmat12
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    starts = oracle.gen_starts(n, g.V, 11)
    paths, lengths = torch.zeros((n, hop), dtype=torch.int32).pin_memory(), torch.zeros(n, dtype=torch.int32).pin_memory()
    kw = dict(app=app, tp=0.1, seed=6, flags=flags)
    _, _, _, edges = ctx.walk(starts, hop, paths=paths, lengths=lengths, **kw)
    want, want_len = np.zeros((n, hop), np.uint32), np.zeros(n, np.uint32)
    _, _, _, want_edges = ctx.walk(starts, hop, paths=want, lengths=want_len, **kw)      # pageable: copied
    assert np.array_equal(lengths.numpy().view(np.uint32), want_len) and edges == want_edges
    assert np.array_equal(paths.numpy().view(np.uint32), want)


@pytest.mark.parametrize("fanout", [[4, 3, 2], [5, 3]])
@pytest.mark.parametrize("per_sm,more", [(6, 0), (6, 1), (8, 0), (8, 1)])
def test_weighted_trees_around_whole_waves(ctx, oracle, rmat12, fanout, per_sm, more):
    """Offline trees of weighted draws have two kernels, chosen by hops and by the CTAs an SM that the batch makes."""
    import torch
    g = rmat12
    n = torch.cuda.get_device_properties(0).multi_processor_count * per_sm + more
    ctx.upload(g.xadj, g.adjncy, g.adjwgt)
    ctx.alias_build_offline()
    table = oracle.alias_build(g.xadj, g.adjwgt)
    seeds = oracle.gen_starts(n, g.V, 4)
    data, sl, _, e = ctx.sample_khop(seeds, fanout, mode=MODE_OFFLINE, seed=5)
    odata, osl = oracle.khop(g.xadj, g.adjncy, g.adjwgt, table, seeds, fanout, seed=5)
    assert np.array_equal(data, odata) and np.array_equal(sl, osl) and e == int(osl.sum())
