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
