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


@pytest.mark.parametrize("w", [4, 8])
def test_a_captured_clean_brings_its_own_scratch(hx, w):
    import torch
    sp, n = 15, 20001
    k, v = workloads.distinct_keys(n, w, 4), workloads.values(n, w, 4)
    dk, dv = _dev(k), _dev(v)
    gone = dk[: n // 4].contiguous()
    out = torch.empty_like(dv)
    fill = int(np.array(FILL, _dt(w)).view(np.int32 if w == 4 else np.int64))
    s = torch.cuda.Stream()
    m = hx.Hashmap(sp, w, stream=s)
    m.insert(dk, dv, target_lf=0.0, stream=s)  # sizes the launch; the map has no scratch yet
    torch.cuda.synchronize()

    def work():
        out.fill_(fill)
        m.clear(stream=s)
        m.insert(dk, dv, target_lf=0.0, stream=s)
        m.erase(gone, stream=s)
        m.clean_tombstones(stream=s)
        m.retrieve(dk, out, stream=s)

    g = _captured(s, work)
    want = v.copy()
    want[: n // 4] = FILL
    for _ in range(3):
        out.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(_host(out, w), want)
        with torch.cuda.stream(s):
            m.clean_tombstones(stream=s)  # eager calls in between use the map's own
            assert m.extract_all_keys(torch.empty(n, dtype=dk.dtype, device="cuda"), stream=s) == n - n // 4
        inf = m.info(stream=s)
        assert (inf.fill, inf.tombstone_counter, inf.err) == (n - n // 4, 0, hx.STATUS_SUCCESS)
    del g
    m.close()


@pytest.mark.parametrize("w", [4, 8])
def test_clean_after_a_replay_keeps_every_key(hx, w):
    import torch
    sp = 15  # several slices: keys whose run crosses a slice's end go through the list
    n = int(0.9 * (1 << sp))
    k, v = workloads.distinct_keys(n, w, 5), workloads.values(n, w, 5)
    dk, dv = _dev(k), _dev(v)
    gone = dk[: n // 3].contiguous()
    s = torch.cuda.Stream()
    m = hx.Hashmap(sp, w, stream=s)
    m.insert(dk, dv, target_lf=0.0, stream=s)
    torch.cuda.synchronize()

    def work():
        m.insert(dk, dv, target_lf=0.0, stream=s)
        m.erase(gone, stream=s)

    g = _captured(s, work)
    m.clear(stream=s)
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    m.clean_tombstones(stream=s)
    out = _dev(np.full(n, FILL, _dt(w)))
    torch.cuda.synchronize()
    m.retrieve(dk, out, stream=s)
    want = v.copy()
    want[: n // 3] = FILL
    inf = m.info(stream=s)
    np.testing.assert_array_equal(_host(out, w), want)
    assert (inf.fill, inf.tombstone_counter, inf.err) == (n - n // 3, 0, hx.STATUS_SUCCESS)
    m.close()


@pytest.mark.parametrize("w", [4, 8])
def test_growth_after_a_replay_counts_its_keys(hx, w):
    import torch
    n = 900
    k, v = workloads.distinct_keys(2 * n, w, 6), workloads.values(2 * n, w, 6)
    dk, dv = _dev(k), _dev(v)
    s = torch.cuda.Stream()
    m = hx.Hashmap(10, w, stream=s)
    m.insert(dk[:n], dv[:n], target_lf=0.0, stream=s)
    torch.cuda.synchronize()
    g = _captured(s, lambda: m.insert(dk[:n], dv[:n], target_lf=0.0, stream=s))
    m.clear(stream=s)
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    m.insert(dk[n:n + 200], dv[n:n + 200], target_lf=0.5, stream=s)  # 1100 keys
    inf = m.info(stream=s)
    assert (inf.fill, inf.err, inf.size_power) == (n + 200, hx.STATUS_SUCCESS, 12)
    m.insert(dk[n + 200:], dv[n + 200:], target_lf=0.5, stream=s)    # 1800 keys: no growth
    out = _dev(np.full(2 * n, FILL, _dt(w)))
    torch.cuda.synchronize()
    m.retrieve(dk, out, stream=s)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(_host(out, w), v)
    assert m.info(stream=s).size_power == 12
    m.close()
