"""Graphs that were captured earlier are replayed between eager calls on the same map:
the eager calls see what the replays did. Integer work: the tolerance is zero."""
import numpy as np
import pytest

from hashinator_gb300 import workloads
from test_bulk_gpu import FILL, _dev, _dt, _host

pytestmark = pytest.mark.gpu


def _captured(s, work):
    import torch
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        work()
    return g


@pytest.mark.parametrize("w", [4, 8])
def test_status_after_a_replay_that_filled_the_table(hx, w):
    import torch
    s = torch.cuda.Stream()
    m = hx.Hashmap(5, w, stream=s)
    k, v = workloads.distinct_keys(40, w, 3), workloads.values(40, w, 3)
    dk, dv = _dev(k), _dev(v)
    m.insert(dk, dv, target_lf=0.0, stream=s)
    torch.cuda.synchronize()
    g = _captured(s, lambda: m.insert(dk, dv, target_lf=0.0, stream=s))
    m.clear(stream=s)
    torch.cuda.synchronize()
    g.replay()  # 40 keys into 32 buckets
    torch.cuda.synchronize()
    assert m.info(stream=s).err == hx.STATUS_FAIL
    m.clear(stream=s)
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    out = _dev(np.full(40, FILL, _dt(w)))
    m.retrieve(dk, out, stream=s)
    torch.cuda.synchronize()
    there = _host(out, w) == v
    assert there.sum() == 32
    at = int(np.nonzero(there)[0][0])
    m.insert(dk[at:at + 1], dv[at:at + 1], target_lf=0.0, stream=s)  # a key that is there: it succeeds
    assert m.peek_status(stream=s) == hx.STATUS_SUCCESS
    m.close()
