"""node2vec's connectivity search at the list shapes where it can go wrong, against the oracle."""
import numpy as np
import pytest

from skywalker_b200 import APP_NODE2VEC, MODE_OFFLINE, WALK_BUILD_TABLES, MODE_ONLINE


def _clustered_graph(V, seed):
    """Lists of 1 .. V - 1 neighbours around the sector size of 8, evenly spread, bunched at either end of the
    id range or in a few runs; every vertex is met again, so searches both hit and miss."""
    rng = np.random.default_rng(seed)
    degs = [1, 2, 7, 8, 9, 15, 16, 17, 31, 33, 64, 100, 257, 1000, V - 1]
    lists = []
    for v in range(V):
        n = degs[v % len(degs)] if v < 300 else degs[rng.integers(0, 10)]
        shape = v % 4
        if shape == 0:
            ids = rng.choice(V, n, replace=False)
        elif shape == 1:
            ids = np.unique((V - 1) * rng.random(n) ** 6)[:n]          # most of them near 0
        elif shape == 2:
            ids = np.unique((V - 1) * (1 - rng.random(n) ** 6))[:n]    # most of them near V
        else:
            base = rng.integers(0, max(1, V - n))
            ids = np.concatenate([np.arange(base, base + n - n // 3), rng.integers(0, V, n // 3)])
        lists.append(np.unique(np.asarray(ids, np.int64)).astype(np.uint32))
    xadj = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.uint32)
    adj = np.concatenate(lists)
    return xadj, adj, rng.uniform(1, 10, len(adj)).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 1, 5])
@pytest.mark.parametrize("p,q", [(2.0, 0.5), (0.5, 2.0), (1.0, 1.0), (100.0, 0.01)])
def test_node2vec_search_shapes(ctx, oracle, shift, p, q):
    import torch
    x, a, w = _clustered_graph(3001, 11)
    V, E = len(x) - 1, len(a)
    d_x = torch.from_numpy(x.view(np.int32)).cuda()
    d_a = torch.zeros(E + 8, dtype=torch.int32, device="cuda")[shift:shift + E]   # borrowed, not on a sector boundary
    d_a.copy_(torch.from_numpy(a.view(np.int32)))
    d_w = torch.from_numpy(w).cuda()
    torch.cuda.synchronize()
    ctx.adopt_device(V, E, d_x, d_a, d_w)
    ctx.alias_build_offline()
    starts = oracle.gen_starts(4000, V, 3)
    want, want_len = oracle.walk(x, a, w, oracle.alias_build(x, w), starts, 31, app=APP_NODE2VEC, p=p, q=q, seed=5)
    live = np.arange(31)[None, :] <= want_len[:, None]
    for mode, flags in ((MODE_OFFLINE, 0), (MODE_ONLINE, 0), (MODE_ONLINE, WALK_BUILD_TABLES)):
        paths, lens, _, edges = ctx.walk(starts, 31, app=APP_NODE2VEC, p=p, q=q, seed=5, mode=mode, flags=flags)
        assert np.array_equal(lens, want_len) and edges == int(want_len.sum())
        assert np.array_equal(paths[live], want[live])


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 3])
@pytest.mark.parametrize("unbiased", [False, True])
@pytest.mark.parametrize("V,share,n,hop", [
    (3001, 1.0, 65, 31), (3001, 1.0, 95000, 31), (3001, 1.0, 222000, 11), (3001, 1.0, 222001, 11),
    (9001, 1.0, 59201, 21), (9001, 1.0, 150000, 17), (9001, 1.0, 150000, 18),
    (9001, 0.7, 88800, 30), (9001, 0.7, 88801, 30), (9001, 0.55, 59201, 20),      # dead ends
    (9001, 0.3, 1, 31), (9001, 0.3, 3000, 31), (9001, 0.3, 3000, 1)])              # ... mostly, short lists
def test_node2vec_kernels(ctx, oracle, shift, unbiased, V, share, n, hop):
    """The node2vec kernels around the sizes that choose between them, with vertices without out-edges."""
    import torch
    x, a, w = _clustered_graph(V, 11)
    deg = np.diff(x.astype(np.int64))
    deg[np.random.default_rng(V).random(V) >= share] = 0
    if share < 0.5:
        deg = np.minimum(deg, 9)
    a = np.concatenate([a[x[v]:x[v] + deg[v]] for v in range(V)])
    w = np.concatenate([w[x[v]:x[v] + deg[v]] for v in range(V)])
    x = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    E = len(a)
    d_a = torch.zeros(E + 8, dtype=torch.int32, device="cuda")[shift:shift + E]   # borrowed, not on a sector boundary
    d_a.copy_(torch.from_numpy(a.view(np.int32)))
    d_x, d_w = torch.from_numpy(x.view(np.int32)).cuda(), torch.from_numpy(w).cuda()
    torch.cuda.synchronize()
    ctx.adopt_device(V, E, d_x, d_a, d_w)
    ctx.alias_build_offline()
    starts = oracle.gen_starts(n, V, 3)
    table = None if unbiased else oracle.alias_build(x, w)
    want, want_len = oracle.walk(x, a, None if unbiased else w, table, starts, hop, app=APP_NODE2VEC, p=0.5, q=2.0, seed=5,
                                 walker_base=9, unbiased=unbiased)
    live = np.arange(hop)[None, :] <= want_len[:, None]
    for mode in (MODE_OFFLINE, MODE_ONLINE):
        paths, lens, _, edges = ctx.walk(starts, hop, app=APP_NODE2VEC, p=0.5, q=2.0, seed=5, walker_base=9, mode=mode,
                                         flags=2 if unbiased else 0)
        assert np.array_equal(lens, want_len) and edges == int(want_len.sum())
        assert np.array_equal(paths[live], want[live])
