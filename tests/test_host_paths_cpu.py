"""Host paths that a GPU takes only when memory is short or streams change, run on the CPU: the library in a child
process whose CUDA runtime is tests/fake_cudart.cpp (no kernel runs; allocations fail on request)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import ctypes as C
import numpy as np
from skywalker_b200 import _capi
from skywalker_b200.api import Context, SkwError
fake = C.CDLL(%r)
fake.fake_log.restype = C.c_char_p
fake.fake_used.restype = C.c_size_t
fake.fake_memory.argtypes = [C.c_size_t]
def calls(clear=True):
    lines = [x.split() for x in fake.fake_log().decode().splitlines()]
    if clear:
        fake.fake_clear_log()
    return lines
def launches(lines, kernel):
    return [x for x in lines if x[0] == "launch" and kernel in x[2]]
class Device:   # stands for a tensor on the device
    is_cuda = True
    def __init__(self, *shape):
        self.a = np.zeros(shape, np.uint32)
    def data_ptr(self):
        return self.a.ctypes.data
    def numel(self):
        return self.a.size
def ring(V=1000, deg=12, hub=0):   # a graph to be resident
    d = np.full(V, deg)
    d[0] += hub
    x = np.concatenate([[0], np.cumsum(d)]).astype(np.uint32)
    return x, np.arange(x[-1], dtype=np.uint32) %% V, np.ones(x[-1], np.float32)
"""


@pytest.fixture(scope="session")
def fake_cudart(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), "-o", out], check=True, timeout=300)
    return out


def _run(fake_cudart, body):
    env = dict(os.environ, LD_PRELOAD=fake_cudart, PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", PRELUDE % fake_cudart + body], capture_output=True, text=True, timeout=300,
                       env=env, cwd=ROOT)
    assert p.returncode == 0, p.stdout + p.stderr


@pytest.mark.parametrize("nth", [0, 1, 2])
@pytest.mark.parametrize("times", [1, 2])
def test_records_build_without_memory(fake_cudart, nth, times):
    """The build of the walk records runs out of memory at any of its three allocations, for good or with one success
    before the next try: an error, no kernel that would write records, and a context that goes on."""
    _run(fake_cudart, """
ctx = Context(0)
ctx.upload(*ring())
ctx.alias_build_offline()
calls()
fake.fake_fail_malloc(%d, %d)
try:
    ctx.walk_records_build()
    assert False, "built"
except SkwError as e:
    assert "out of memory" in str(e), e
assert not [x for x in calls() if x[0] == "launch"]
fake.fake_fail_malloc(-1, 0)
ctx.walk_records_build()
assert launches(calls(), "walk_records_kernel")
ctx.walk_records_build()
log = calls()
assert launches(log, "walk_records_kernel") and not [x for x in log if x[0] == "malloc"]
""" % (nth, times))


def test_records_that_wait_for_a_rebuild_make_room(fake_cudart):
    """Records of a table that was built anew are given up when another allocation fails."""
    _run(fake_cudart, """
ctx = Context(0)
ctx.upload(*ring())
ctx.alias_build_offline()
ctx.walk_records_build()
ctx.alias_build_offline()
calls()
fake.fake_fail_malloc(0, 1)
ctx.walk(np.zeros(5000, np.uint32), 50)      # its staging buffers are new
log = calls()
assert sum(x[0] == "malloc" and x[2] == "fail" for x in log) == 1
assert sum(x[0] == "device_sync" for x in log) >= 3    # three blocks returned
""")


@pytest.mark.parametrize("call", ["walk", "walk_packed"])
def test_online_tables_are_built_once_a_call(fake_cudart, call):
    """Large batches with host results run in slices; the tables of the whole graph serve all of them."""
    _run(fake_cudart, """
ctx = Context(0)
ctx.upload(*ring())
calls()
n = (1 << 21) + 5          # four slices
starts = np.zeros(n, np.uint32)
try:
    ctx.%s(starts, 3, mode=1)
except SkwError as e:      # (no kernel ran, so the rows do not add up)
    assert "lengths add up" in str(e), e
log = calls()
assert len(launches(log, "walk_offline_kernel")) == 4 and not launches(log, "direct")
assert len(launches(log, "classify_kernel")) == 1
""" % call)


@pytest.mark.parametrize("nth,times,hub", [(0, 1, 0), (1, 1, 0), (2, 1, 0), (0, 1000, 0), (2, 1000, 0), (3, 1, 20000)])
def test_online_walk_without_memory_for_tables(fake_cudart, nth, times, hub):
    """Tables of the whole graph are a choice of the library: where their memory (slots, flags, work lists, scratch of
    the longest lists) is not to be had, the walk computes its slots one by one."""
    _run(fake_cudart, """
ctx = Context(0)
ctx.upload(*ring(hub=%d))
s, p, l = Device(1 << 18), Device(1 << 18, 20), Device(1 << 18)
calls()
fake.fake_fail_malloc(%d, %d)
ctx.walk(s, 20, mode=1, paths=p, lengths=l)
log = calls()
assert sum(x[0] == "malloc" and x[2] == "fail" for x in log)
assert len(launches(log, "walk_online_direct_kernel")) == 1 and not launches(log, "classify")
fake.fake_fail_malloc(-1, 0)
ctx.walk(s, 20, mode=1, paths=p, lengths=l)
log = calls()
assert len(launches(log, "classify")) == 1 and len(launches(log, "walk_offline_kernel")) == 1
""" % (hub, nth, times))


def test_tables_of_an_online_call_make_room(fake_cudart):
    """The memory of an online call's tables is kept for the next one, but given up when an allocation fails without it,
    and returned with the weights."""
    _run(fake_cudart, """
ctx = Context(0)
V, E = 40000, 480000
ctx.upload(*ring(V))
s, p, l = Device(1 << 18), Device(1 << 18, 20), Device(1 << 18)
ctx.walk(s, 20, mode=1, paths=p, lengths=l)
calls()
fake.fake_memory(fake.fake_used() + 8 * E - 1)      # room for nearly the table
ctx.alias_build_offline()
ctx.walk(s, 20, mode=1, paths=p, lengths=l)         # nothing left for tables of its own
log = calls()
assert len(launches(log, "walk_online_direct_kernel")) == 1
fake.fake_memory(64 << 30)
ctx.walk(s, 20, mode=1, paths=p, lengths=l)
assert len(launches(calls(), "walk_offline_kernel")) == 1
used = fake.fake_used()
ctx.free_weights()
assert used - fake.fake_used() >= 4 * E + 8 * E
""")


@pytest.mark.parametrize("warm", [None, 256, 1 << 18])
@pytest.mark.parametrize("hub", [0, 20000])
def test_online_walk_under_capture_allocates_nothing(fake_cudart, warm, hub):
    """A queued online walk can be captured into a graph, whatever ran before it: one kernel, and no memory that the
    library may later take away from the graph."""
    _run(fake_cudart, """
ctx = Context(0)
ctx.upload(*ring(hub=%d))
s, p, l = Device(1 << 18), Device(1 << 18, 20), Device(1 << 18)
if %r:
    ctx.walk(s, 20, mode=1, paths=p, lengths=l, n=%r)
calls()
fake.fake_capture(1)
ctx.walk(s, 20, mode=1, paths=p, lengths=l, enqueue_only=True)
log = calls()
assert len(log) == 1 and launches(log, "walk_online_direct_kernel"), log
fake.fake_capture(0)
ctx.walk(s, 20, mode=1, paths=p, lengths=l, enqueue_only=True)
assert launches(calls(), "walk_offline_kernel")
""" % (hub, warm, warm))


@pytest.mark.parametrize("flags", [0, 4])       # tables of the whole graph, of every step's vertices
@pytest.mark.parametrize("then", ["build", "queued", "khop"])
def test_builders_wait_for_queued_tables_on_another_stream(fake_cudart, flags, then):
    """Work lists, scratch and online tables belong to the context: after a change of stream a call that builds tables
    waits for queued walks that still use them."""
    _run(fake_cudart, """
ctx = Context(0)
ctx.upload(*ring(hub=20000))
ctx.alias_build_offline()
s, p, l = Device(1 << 18), Device(1 << 18, 20), Device(1 << 18)
one, two = C.create_string_buffer(8), C.create_string_buffer(8)
ctx.set_stream(C.addressof(one))
calls()
ctx.walk(s, 20, mode=1, paths=p, lengths=l, flags=%d, enqueue_only=True)
first = calls()
ctx.set_stream(C.addressof(two))
if %r == "build":
    ctx.alias_build_offline()
elif %r == "khop":
    ctx.sample_khop(np.zeros(100, np.uint32), [5, 3], mode=1)
else:
    ctx.walk(s, 20, mode=1, paths=p, lengths=l, enqueue_only=True)
second = calls()
# what the last kernel of the first call happens before, through stream order and events
a, b = hex(C.addressof(one)), hex(C.addressof(two))
last = max(i for i, x in enumerate(first) if x[0] == "launch" and x[1] == a)
reached, events = {a}, set()
builders = 0
for x in first[last + 1:] + second:
    if x[0] == "record":
        (events.add if x[2] in reached else events.discard)(x[1])
    elif x[0] == "wait" and x[2] in events:
        reached.add(x[1])
    elif x[0] == "device_sync":
        reached.update((a, b))
    elif x[0] in ("launch", "memset") and (x[0] == "memset" or any(k in x[2] for k in ("classify", "collect", "build_"))):
        builders += 1
        assert x[1] in reached, (x, reached)
assert builders > 3
""" % (flags, then, then))


@pytest.mark.parametrize("writer", ["alias_build_offline()", "alias_build_offline(0, 10)", "walk_records_build()", "alias_load(path)",
                                    "alias_import(*table)"])
def test_table_writers_wait_for_queued_walks_on_another_stream(fake_cudart, tmp_path, writer):
    """A table or its records are written in place; walks that were queued on another stream may still read them."""
    _run(fake_cudart, """
path = %r
ctx = Context(0)
ctx.upload(*ring())
ctx.alias_build_offline()
ctx.alias_save(path)
table = ctx.alias_export()
ctx.walk_records_build()
s, p, l = Device(1 << 10), Device(1 << 10, 20), Device(1 << 10)
one, two = C.create_string_buffer(8), C.create_string_buffer(8)
ctx.set_stream(C.addressof(one))
ctx.walk(s, 20, paths=p, lengths=l, enqueue_only=True)
ctx.set_stream(C.addressof(two))
calls()
ctx.%s
assert calls()[0] == ["device_sync"]
ctx.%s
assert ["device_sync"] not in calls()       # once
ctx.walk(s, 20, paths=p, lengths=l, enqueue_only=True)
ctx.%s                                      # the same stream: its order is enough
assert ["device_sync"] not in calls()
""" % (str(tmp_path / "t.skw"), writer, writer, writer))


@pytest.mark.parametrize("times", [1, 1000])
def test_results_without_pinned_memory(fake_cudart, times):
    """Result arrays come from pinned memory where there is some, else from pageable memory."""
    _run(fake_cudart, """
ctx = Context(0)
ctx.upload(*ring())
ctx.alias_build_offline()
calls()
fake.fake_fail_host_malloc(0, %d)
for _ in range(3):
    paths, lengths, _, _ = ctx.walk(np.zeros(100, np.uint32), 5)
    assert paths.shape == (100, 5) and lengths.shape == (100,)
assert sum(x[0] == "host_malloc" and x[1] == "fail" for x in calls()) >= 1
""" % times)


@pytest.mark.parametrize("call", ["alias_build_offline()", "sample_khop(np.zeros(10, np.uint32), [3], mode=1)",
                                  "walk(np.zeros(5000, np.uint32), 100, flags=2)"])
@pytest.mark.parametrize("after", [0, 2])
def test_call_after_one_that_ran_out_of_memory(fake_cudart, call, after):
    """An error that a call has reported is not met again by the next one."""
    _run(fake_cudart, """
ctx = Context(0)
ctx.upload(*ring())
fake.fake_fail_malloc(%d, 1000)
try:
    ctx.%s
    assert False
except SkwError as e:
    assert "out of memory" in str(e) and "dev_malloc" in str(e), e
fake.fake_fail_malloc(-1, 0)
ctx.%s
""" % (after, call, call))


@pytest.mark.parametrize("n", [1000, 1 << 18])
def test_refused_walk_leaves_the_rows_alone(fake_cudart, n):
    _run(fake_cudart, """
ctx = Context(0)
ctx.upload(*ring())
paths, lengths = np.full((%d, 3), 5, np.uint32), np.full(%d, 5, np.uint32)
try:                                   # 16: fill the rows; there is no table
    ctx.walk(np.zeros(%d, np.uint32), 3, paths=paths, lengths=lengths, flags=16)
    assert False
except SkwError as e:
    assert e.code == -3
assert (paths == 5).all() and (lengths == 5).all()
""" % (n, n, n))


def test_rows_are_written_home_only_where_they_are_filled(fake_cudart):
    """Without the flag that fills the rows no row is written before the whole batch is known to be good."""
    _run(fake_cudart, """
fake.fake_pinned(1)
ctx = Context(0)
ctx.upload(*ring())
ctx.alias_build_offline()
from skywalker_b200.api import _results
paths, lengths = _results.array((300, 81)), _results.array((300,))
for app in (0, 1):
    for unbiased in (0, 2):
        for fill in (0, 16):
            calls()
            ctx.walk(np.zeros(300, np.uint32), 81, app=app, tp=0.15, paths=paths, lengths=lengths, flags=unbiased | fill)
            log = calls()
            assert len(launches(log, "walk_home_kernel")) == (fill != 0), log
            assert len(launches(log, "walk_offline_kernel")) == (fill == 0), log
""")


@pytest.mark.parametrize("ends,app,tp,n,hop,home", [
    (False, 0, 0.0, 29600, 201, True), (False, 0, 0.0, 4096, 1001, True), (False, 0, 0.0, 29601, 81, False),
    (False, 0, 0.0, 5032, 32, True), (False, 0, 0.0, 5033, 32, False), (True, 0, 0.0, 4096, 81, True),
    (True, 0, 0.0, 29600, 81, False), (True, 0, 0.0, 29600, 33, False), (True, 0, 0.0, 256, 161, False),
    (False, 1, 0.15, 4096, 201, True), (False, 1, 0.15, 29600, 81, True), (True, 1, 0.15, 29600, 81, False),
    (False, 1, 0.15, 29600, 201, False), (False, 1, 0.15, 10000, 501, False), (False, 1, 0.15, 256, 1001, False),
    (False, 1, 0.0, 4096, 1001, True), (False, 1, 1.0, 4096, 101, True), (False, 1, 1.0, 10000, 101, False)])
def test_rows_are_written_home_where_walks_hide_it(fake_cudart, ends, app, tp, n, hop, home):
    """Walks hide the writes only while they last; matrices whose cells mostly lie behind the ends of all walks are copied."""
    _run(fake_cudart, """
fake.fake_pinned(1)
ctx = Context(0)
x, a, w = ring()
if %r:                                  # every edge leads to a vertex without out-edges
    x = np.concatenate([x, np.full(10, x[-1])]).astype(np.uint32)
    a[:] = 1000
ctx.upload(x, a, w)
ctx.alias_build_offline()
calls()
ctx.walk(np.zeros(%d, np.uint32), %d, app=%d, tp=%g)
log = calls()
assert len(launches(log, "walk_home_kernel")) == %d and len(launches(log, "walk_offline_kernel")) == %d
""" % (ends, n, hop, app, tp, home, not home))


@pytest.mark.parametrize("call", ["alias_build_offline()", "walk(s, 20, mode=1, paths=p, lengths=l)",
                                  "sample_khop(np.zeros(2000, np.uint32), [5, 3], mode=1)"])
def test_long_lists_without_memory_for_small_teams(fake_cudart, call):
    """Lists of more than 16384 weights beyond what teams of eight CTAs take at a time go to smaller teams, with more
    scratch; without memory for that the teams of eight take them all."""
    _run(fake_cudart, """
def context():
    ctx = Context(0)
    d = np.full(1000, 12)
    d[:60] = 20000
    x = np.concatenate([[0], np.cumsum(d)]).astype(np.uint32)
    ctx.upload(x, np.arange(x[-1], dtype=np.uint32) %% 1000, np.ones(x[-1], np.float32))
    return ctx
MB = 1 << 20
s, p, l = Device(1 << 18), Device(1 << 18, 20), Device(1 << 18)
ctx = context()
idle = fake.fake_used()
ctx.%s
log = calls()
need = fake.fake_used() - idle
assert need > 110 * MB and launches(log, "build_long_kernelILj4E") and not launches(log, "direct")
ctx.close()
ctx = context()
fake.fake_memory(fake.fake_used() + need - 60 * MB)
for _ in range(2):
    ctx.%s
    log = calls()
    assert launches(log, "build_long_kernelILj8E") and not launches(log, "build_long_kernelILj4E")
assert not [x for x in log if x[0] == "malloc"]
ctx.close()
# without memory for either the call fails (walks compute their slots), and the next one has all of it
ctx = context()
fake.fake_memory(fake.fake_used() + 4 * MB)
try:
    ctx.%s
    assert launches(calls(), "direct")
except SkwError as e:
    assert "out of memory" in str(e)
fake.fake_memory(64 << 30)
calls()
ctx.%s
assert launches(calls(), "build_long_kernelILj4E")
ctx.upload(*ring(hub=20000))
ctx.alias_build_offline()
assert ctx.alias_export()[0].size == 32000
""" % (call, call, call, call))


def test_rows_of_which_only_parts_are_registered_are_copied(fake_cudart):
    """The GPU writes a matrix of the caller's only if all of it is one pinned range: not one whose ends are pinned, with
    other pages between them, or one that ends behind the range."""
    _run(fake_cudart, """
fake.fake_pinned(1)
fake.fake_register.argtypes = [C.c_void_p, C.c_size_t]
ctx = Context(0)
ctx.upload(*ring())
ctx.alias_build_offline()
lengths = np.zeros(300, np.uint32)
fake.fake_register(lengths.ctypes.data, lengths.nbytes)
for parts, home in (([(0, 4096), (93104, 4096)], 0), ([(0, 97196)], 0), ([(4, 97196)], 0), ([(0, 97200)], 1)):
    paths = np.zeros((300, 81), np.uint32)
    for at, size in parts:
        fake.fake_register(paths.ctypes.data + at, size)
    calls()
    ctx.walk(np.zeros(300, np.uint32), 81, paths=paths, lengths=lengths, flags=16)
    assert len(launches(calls(), "walk_home_kernel")) == home, parts
    globals().setdefault("keep", []).append(paths)      # (the addresses stay taken)
""")


@pytest.mark.parametrize("V,ends,fanout,n,more", [
    (1000, 0, [25, 10], 888, False), (1000, 0, [25, 10], 889, True), (1000, 0, [25, 10], 1184, True), (1000, 0, [25, 10], 1300, False),
    (1000, 0, [25, 10], 2000, True), (1000, 0, [25, 10], 20000, False), (200000, 0, [25, 10], 20000, True),
    (200000, 0, [25, 10], 13645, False), (400000, 0, [10, 5], 13645, False), (400000, 200000, [10, 5], 13645, True),
    (400000, 200000, [25, 10], 13645, False), (1000, 0, [40], 65536, True), (1000, 0, [15, 10, 5], 1000, True),
    (400000, 0, [15, 10, 5], 2000, False)])
def test_warps_of_weighted_trees(fake_cudart, V, ends, fanout, n, more):
    """Which of its two kernels a batch of trees takes: eight CTAs an SM where they save a wave and the tables are large."""
    _run(fake_cudart, """
ctx = Context(0)
x, a, w = ring(%d)
ctx.upload(np.concatenate([x, np.full(%d, x[-1])]).astype(np.uint32), a, w)
ctx.alias_build_offline()
cells, lens = ctx.khop_layout(%r)
calls()
ctx.sample_khop(Device(%d), %r, mode=0, data=Device(%d, cells), sample_lengths=Device(%d, lens))
log = calls()
assert len(launches(log, "khop_weighted_tree_kernel")) == %d and len(launches(log, "khop_tree_kernelILb0")) == %d
""" % (V, ends, fanout, n, fanout, n, n, more, not more))


@pytest.mark.parametrize("V,n,hop,ahead", [(1000, 5920, 17, True), (1000, 5921, 17, False), (1000, 39000, 40, False),
                                           (1000, 39000, 41, True), (60000, 39000, 17, True), (60000, 39961, 17, False)])
def test_ppr_neighbours_beside_their_slots(fake_cudart, V, n, hop, ahead):
    """Which kernel walks over slots take: the one that fetches neighbours ahead is for walks that wait for memory."""
    _run(fake_cudart, """
ctx = Context(0)
ctx.upload(*ring(%d))
ctx.alias_build_offline()
s, p, l = Device(%d), Device(%d, %d), Device(%d)
calls()
ctx.walk(s, %d, app=1, tp=0.15, paths=p, lengths=l)
assert len(launches(calls(), "walk_offline_kernelILi1ELb%dE")) == 1
""" % (V, n, n, hop, n, hop, ahead))


def test_packed_ppr_without_memory_for_heads(fake_cudart):
    """The first cells of the rows travel apart from them where there is memory: it is asked for behind everything that
    the call needs, and given up when another allocation fails, also in the middle of a call."""
    _run(fake_cudart, """
n, hop, MB = 200000, 101, 1 << 20
kw = dict(app=1, tp=0.15)
def context():
    ctx = Context(0)
    ctx.upload(*ring())
    ctx.alias_build_offline()
    ctx.walk_records_build()
    ctx.walk(np.zeros(10, np.uint32), 5)
    calls()
    return ctx
starts, packed, lengths = np.zeros(n, np.uint32), np.zeros(4000000, np.uint32), np.zeros(n, np.uint32)
def walk(ctx):
    used = fake.fake_used()
    ctx.walk_packed(starts, hop, packed=packed, lengths=lengths, **kw)
    log = calls()
    return len(launches(log, "pack_heads")), len(launches(log, "pack_rows")), (fake.fake_used() - used) / MB
ctx = context()
heads, rows, need = walk(ctx)
assert (heads, rows) == (1, 0) and need > 90
ctx.close()
# two megabytes less than all of it: enough without the heads
ctx = context()
fake.fake_memory(int(fake.fake_used() + (need - 2) * MB))
assert walk(ctx)[:2] == (0, 1)
fake.fake_memory(64 << 30)
assert walk(ctx)[:2] == (1, 0)
# kept for the next call, given up for another allocation
fake.fake_memory(fake.fake_used() + MB)
assert walk(ctx)[:2] == (1, 0)
n += 10000                       # four megabytes of rows more
starts, lengths = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
assert walk(ctx)[:2] == (0, 1)
fake.fake_memory(64 << 30)
assert walk(ctx)[:2] == (1, 0)
# a result that outgrows its buffer in a call that holds the heads
fake.fake_memory(fake.fake_used() + MB)
fake.fake_packed(3600000)
assert walk(ctx)[:2] == (1, 2)
fake.fake_memory(64 << 30)
assert walk(ctx)[:2] == (1, 0)
""")


def test_freed_device_memory_waits_within_bounds(fake_cudart):
    """Freed blocks serve the next graph, up to a sixteenth of the memory, and are returned when an allocation fails
    without them, on request, and with the last context."""
    _run(fake_cudart, """
G = 1 << 30
fake.fake_memory(16 * G)
idle = fake.fake_used()
a, b = Context(0), Context(0)
a.upload(*ring(100000))
a.alias_build_offline()
calls()
a.upload(*ring(100000))
a.alias_build_offline()
log = calls()
assert not [x for x in log if x[0] == "malloc"]            # the same sizes again
free = [i for i, x in enumerate(log) if x[0] == "device_sync"]
assert free and free[0] < min(i for i, x in enumerate(log) if x[0] in ("copy", "launch"))   # idle before it is used again
for v in (300000, 500000, 700000, 900000, 1100000, 1500000, 2000000):
    a.upload(*ring(v))
    a.alias_build_offline()
    a.walk_records_build()
    live = v * 12 * (8 + 8 + 32) + v * 24
    assert fake.fake_used() - live < G + (64 << 20) + v * 300, (v, fake.fake_used() >> 20)   # a sixteenth, and the work lists
held = fake.fake_used()
a.walk_records_free()
assert fake.fake_used() <= held - 2000000 * 12 * 32
a.upload(*ring(1000))
waiting = fake.fake_used()
fake.fake_memory(waiting + (1 << 20))                      # an allocation of more than is unused
a.upload(*ring(300000))
fake.fake_memory(16 * G)
a.close()
b.close()
assert fake.fake_used() == idle
""")


def test_result_pool_lends_within_bounds(fake_cudart):
    """Pinned result arrays: a block serves again when the last view of it is gone, so many bytes are out or wait at a
    time, and large results are pageable."""
    _run(fake_cudart, """
import gc, threading
from skywalker_b200 import api
pool = api._results
def pinned(n):
    return sum(x[0] == "host_malloc" for x in calls()) == n
calls()
x = pool.array((1000, 10))
at = x.ctypes.data
view = x[3:7].T
assert pinned(1)
del x
y = pool.array((1000, 10))                 # the first block is still seen through a view
assert pinned(1) and y.ctypes.data != at
del view
gc.collect()
z = pool.array((500, 17))                  # the same size class
assert pinned(0) and z.ctypes.data == at
big = pool.array((pool.LARGEST // 4 + 1,))
assert pinned(0) and big.flags.owndata
out = [pool.array((pool.LARGEST // 4,)) for _ in range(8)]
assert sum(not a.flags.owndata for a in out) == 3 and pool.out <= pool.OUT     # beside y and z
del out, y, z
gc.collect()
assert pool.out == 0 and pool.kept <= pool.KEEP
assert sum(len(v) * k for k, v in pool.waiting.items()) == pool.kept
# threads: no block is lent twice
seen, bad = set(), []
lock = threading.Lock()
def work():
    for _ in range(300):
        a = pool.array((700,))
        with lock:
            (bad.append if a.ctypes.data in seen else seen.add)(a.ctypes.data)
        a[:] = 1
        with lock:
            seen.discard(a.ctypes.data)
        del a
ts = [threading.Thread(target=work) for _ in range(8)]
[t.start() for t in ts]
[t.join() for t in ts]
assert not bad and pool.out == 0 and pool.kept <= pool.KEEP
""")
