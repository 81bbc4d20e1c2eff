"""Tables at the edges of every degree class, for weights at the edges of the arithmetic, against the oracle."""
import numpy as np
import pytest

SIZES = sorted({max(1, b + d) for b in (1, 8, 16, 32, 64, 128, 256, 512, 1024, 2048, 4096, 8192, 16384) for d in (-1, 0, 1)}
               | {3, 100, 300, 777, 1500, 3000, 5000, 12000, 20001, 40000})


def _weights(kind, n, rng):
    if kind == "uniform":
        return rng.uniform(1, 10, n)
    if kind == "equal":
        return np.full(n, 3.0)
    if kind == "one_heavy":           # nearly all mass in one bucket
        w = np.full(n, 1e-6)
        w[rng.integers(0, n)] = 1e6
        return w
    if kind == "one_light":           # many larges, each a little over a bucket
        w = np.ones(n)
        w[rng.integers(0, n)] = 1e-7
        return w
    if kind == "lognormal":
        return rng.lognormal(0, 3, n)
    if kind == "pareto":
        return rng.pareto(0.5, n) + 1e-3
    if kind == "tiny":                # largest weight below 2^-87, denormals among them
        return rng.uniform(0, 1, n) * 10.0 ** rng.integers(-45, -30, n)
    if kind == "unusable":            # zeros, negatives, infinities and NaNs between usable ones, zeros at the end
        w = rng.uniform(1, 10, n)
        w[rng.random(n) < 0.3] = 0.0
        for x in (-1.0, -0.0, np.inf, -np.inf, np.nan):
            w[rng.random(n) < 0.05] = x
        w[n - n // 5:] = 0.0
        return w
    raise ValueError(kind)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["uniform", "equal", "one_heavy", "one_light", "lognormal", "pareto", "tiny", "unusable"])
@pytest.mark.parametrize("shift", [0, 3])
def test_alias_class_edges(ctx, oracle, kind, shift):
    import torch
    rng = np.random.default_rng(len(kind) + shift)
    sizes = SIZES + [2, 5, 300, 900]
    x = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    E = int(x[-1])
    V = len(sizes)
    with np.errstate(over="ignore"):
        w = np.concatenate([_weights(kind, n, rng) for n in sizes]).astype(np.float32)
    a = np.concatenate([np.arange(n) % V for n in sizes]).astype(np.uint32)
    d_w = torch.zeros(E + 4, device="cuda")[shift:shift + E]      # borrowed, not on a 16-byte boundary
    d_w.copy_(torch.from_numpy(w))
    d_x, d_a = (torch.from_numpy(v.view(np.int32)).cuda() for v in (x, a))
    torch.cuda.synchronize()
    ctx.adopt_device(V, E, d_x, d_a, d_w)
    ctx.alias_build_offline()
    prob, alias, valid = ctx.alias_export()
    want_prob, want_alias, want_valid = oracle.alias_build(x, w)
    assert np.array_equal(valid, want_valid)
    usable = np.repeat(want_valid.astype(bool), sizes)
    bad = np.flatnonzero(usable & ((prob != want_prob) | (alias != want_alias)))
    assert bad.size == 0, "list lengths that differ: %s" % sorted({sizes[np.searchsorted(x, b, "right") - 1] for b in bad})


@pytest.mark.gpu
@pytest.mark.parametrize("least, most, lists", [(513, 1024, 3000), (1025, 2048, 1500), (2049, 4096, 700), (1, 40, 200000), (3, 4500, 1500)])
def test_alias_several_lists_a_worker(ctx, oracle, least, most, lists):
    """More lists of a class than there are lanes, warps or parts of a CTA to take one each, next to few of the others."""
    import torch
    rng = np.random.default_rng(most)
    sizes = np.concatenate([rng.integers(least, most + 1, lists), [0, 7, 20, 90, 700, 1300, 3000, 9000, 17000]])
    rng.shuffle(sizes)
    x = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    E, V = int(x[-1]), len(sizes)
    w = rng.lognormal(0, 1, E).astype(np.float32)
    d_x, d_a = torch.from_numpy(x.view(np.int32)).cuda(), torch.zeros(E, dtype=torch.int32, device="cuda")
    d_w = torch.from_numpy(w).cuda()
    torch.cuda.synchronize()
    ctx.adopt_device(V, E, d_x, d_a, d_w)
    ctx.alias_build_offline()
    prob, alias, valid = ctx.alias_export()
    want_prob, want_alias, want_valid = oracle.alias_build(x, w)
    assert np.array_equal(valid, want_valid) and np.array_equal(prob, want_prob) and np.array_equal(alias, want_alias)


KINDS = ["uniform", "equal", "one_heavy", "one_light", "lognormal", "pareto", "tiny", "unusable"]


def _check_lists(ctx, oracle, lists):
    import torch
    sizes = [len(w) for w in lists]
    x = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    with np.errstate(over="ignore"):
        w = np.concatenate(lists).astype(np.float32)
    d_x, d_a = torch.from_numpy(x.view(np.int32)).cuda(), torch.zeros(len(w), dtype=torch.int32, device="cuda")
    d_w = torch.from_numpy(w).cuda()
    torch.cuda.synchronize()
    ctx.adopt_device(len(sizes), len(w), d_x, d_a, d_w)
    ctx.alias_build_offline()
    prob, alias, valid = ctx.alias_export()
    want_prob, want_alias, want_valid = oracle.alias_build(x, w)
    assert np.array_equal(valid, want_valid)
    usable = np.repeat(want_valid.astype(bool), sizes)
    bad = np.flatnonzero(usable & ((prob != want_prob) | (alias != want_alias)))
    assert bad.size == 0, "list lengths that differ: %s" % sorted({sizes[np.searchsorted(x, b, "right") - 1] for b in bad})


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("more_than_clusters", [-1, 0, 1, 150])
def test_alias_many_giant_lists(ctx, oracle, kind, more_than_clusters):
    """Lists of more than 16384 weights of all kinds by teams of eight CTAs, by teams of four from one list more than there are
    teams of eight on, and by pairs, with a list without usable weights between others."""
    import torch
    rng = np.random.default_rng(len(kind))
    clusters = torch.cuda.get_device_properties(0).multi_processor_count * 3 // 8
    sizes = [16385, 16386, 20000, 24575, 24576, 24577, 32768, 32769, 40000, 16384 + 2048, 16384 + 2049]
    sizes = [sizes[i % len(sizes)] for i in range(clusters + more_than_clusters)]
    lists = [_weights(kind, n, rng) for n in sizes]
    lists[len(lists) // 2] = np.zeros(sizes[len(lists) // 2])
    _check_lists(ctx, oracle, lists)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["lognormal", "one_heavy"])
@pytest.mark.parametrize("others", [0, 60])
def test_alias_list_of_many_windows(ctx, oracle, kind, others):
    """A list that takes more than one round of merge windows, alone and behind others that take more teams than there are of
    eight CTAs: a list of more than 65536 weights always has a team of eight."""
    rng = np.random.default_rng(others)
    _check_lists(ctx, oracle, [_weights(kind, 20000, rng) for _ in range(others)] + [_weights(kind, 1024 * 8192 + 5, rng)])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["uniform", "one_heavy", "unusable"])
def test_alias_many_lists_of_one_tile(ctx, oracle, kind):
    """Lists of 4097 to 16384 weights, more of them than CTAs take at a time, around whole numbers of weights a thread; a
    list without usable weights is the last, the first and one between."""
    import torch
    rng = np.random.default_rng(len(kind))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    edges = [4097, 4608, 4609, 5000, 7680, 7681, 8191, 8192, 8193, 9216, 9217, 12000, 15360, 15361, 16383, 16384]
    sizes = edges + list(rng.integers(4097, 8193, 2 * sms)) + list(rng.integers(8193, 16385, sms))
    rng.shuffle(sizes)
    lists = [_weights(kind, n, rng) for n in sizes]
    for i in (0, len(sizes) // 2, len(sizes) - 1):
        lists[i] = np.zeros(sizes[i])
    _check_lists(ctx, oracle, lists)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["uniform", "one_heavy"])
@pytest.mark.parametrize("quarters", [1, 2])
@pytest.mark.parametrize("more", [0, 1])
def test_alias_teams_of_long_lists(ctx, oracle, kind, quarters, more):
    """Lists of 16385 to 65536 weights by fours, pairs and single CTAs, at the counts where the teams change, next to longer
    ones; all vertices at once, and in two ranges, whose kernels find the number of lists for themselves."""
    import torch
    rng = np.random.default_rng(quarters)
    ctas = torch.cuda.get_device_properties(0).multi_processor_count * 3
    sizes = [16385 + (i * 977) % 3000 for i in range(ctas * quarters // 4 + more - 2)] + [65535, 65536] + [65537, 100001]
    lists = [_weights(kind, n, rng) for n in sizes]
    lists[len(lists) // 2] = np.zeros(sizes[len(lists) // 2])
    _check_lists(ctx, oracle, lists)
    whole = ctx.alias_export()
    cut = len(lists) // 3
    ctx.alias_build_offline(0, cut)
    ctx.alias_build_offline(cut, len(lists))
    assert all(np.array_equal(a, b) for a, b in zip(whole, ctx.alias_export()))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["uniform", "one_heavy", "unusable"])
@pytest.mark.parametrize("team", [8, 4, 2, 1])
def test_alias_edges_of_tiles_and_windows(ctx, oracle, kind, team):
    """Lists around whole numbers of tiles of 4096 weights a CTA, chunks that end in few weights, and merge windows of whole and of
    other sizes, by teams of each size."""
    import torch
    ctas = torch.cuda.get_device_properties(0).multi_processor_count * 3
    rng = np.random.default_rng(team)
    sizes = [team * t * 4096 + d for t in (1, 2, 3, 5) for d in (-257, -256, -1, 0, 1, 255, 256, 257)]
    sizes += [team * 256 * k + d for k in (9, 15, 17, 33, 65) for d in (0, 1)] + [65535]
    sizes = [n for n in sizes if 16384 < n <= 65536]
    while len(sizes) <= {8: 0, 4: ctas // 8, 2: ctas // 4, 1: ctas // 2 + ctas // 6}[team]:
        sizes.append(16385 + len(sizes))
    assert len(sizes) <= {8: ctas // 8, 4: ctas // 4, 2: ctas // 2, 1: ctas}[team]
    _check_lists(ctx, oracle, [_weights(kind, n, rng) for n in sizes])


@pytest.mark.gpu
@pytest.mark.parametrize("part, more", [(8, 0), (8, 1), (6, 0), (6, 1)])
def test_alias_more_long_lists_than_pairs(ctx, oracle, part, more):
    """A few lists of 16385 to 65536 weights more than there are pairs of CTAs go to teams of eight or four, which may be at
    work beside the pairs; at the counts where that changes, all vertices at once and in two ranges."""
    import torch
    ctas = torch.cuda.get_device_properties(0).multi_processor_count * 3
    rng = np.random.default_rng(part)
    lists = [_weights("uniform", 16385 + (i * 977) % 2000, rng) for i in range(ctas // 2 + ctas // part + more)]
    lists[5] = _weights("one_heavy", 65536, rng)
    lists[-1] = np.zeros(20000)
    _check_lists(ctx, oracle, lists)
    whole = ctx.alias_export()
    ctx.alias_build_offline(0, 40)
    ctx.alias_build_offline(40, len(lists))
    assert all(np.array_equal(a, b) for a, b in zip(whole, ctx.alias_export()))


@pytest.mark.gpu
@pytest.mark.parametrize("before, after", [(60, 20), (20, 60), (240, 20), (20, 240)])
def test_alias_offsets_of_a_borrowed_graph_change(ctx, oracle, before, after):
    """The offsets of a borrowed graph are rewritten in place: another number of lists of 16385 to 65536 weights than the
    teams were launched for.  All of them are built."""
    import torch
    E = 65536 + 240 * 16385
    def offsets(lists):
        sizes = [65536] + [16385 * (240 // lists) if 16385 * (240 // lists) <= 65536 else 49155] * lists
        sizes += [1000] * 240
        sizes[-240:] = [(E - sum(sizes[:-240])) // 240] * 239 + [(E - sum(sizes[:-240])) // 240 + (E - sum(sizes[:-240])) % 240]
        assert sum(sizes) == E and all(n <= 16384 for n in sizes[-240:])
        sizes += [0] * (500 - len(sizes))
        return np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    w = np.random.default_rng(before).uniform(1, 10, E).astype(np.float32)
    x = torch.from_numpy(offsets(before).view(np.int32)).cuda()
    a, d_w = torch.zeros(E, dtype=torch.int32, device="cuda"), torch.from_numpy(w).cuda()
    torch.cuda.synchronize()
    ctx.adopt_device(500, E, x, a, d_w)
    ctx.alias_build_offline()
    x.copy_(torch.from_numpy(offsets(after).view(np.int32)))
    torch.cuda.synchronize()
    for ranges in ([(0, 500)], [(0, 100), (100, 500)]):
        for r in ranges:
            ctx.alias_build_offline(*r)
        prob, alias, valid = ctx.alias_export()
        want_prob, want_alias, want_valid = oracle.alias_build(offsets(after), w)
        assert np.array_equal(valid, want_valid) and np.array_equal(prob, want_prob) and np.array_equal(alias, want_alias)
