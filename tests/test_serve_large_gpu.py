"""One request of many more keys than the server's rounds are meant for: it runs as a
round of its own, with exact results. Integer work: the tolerance is zero."""
import numpy as np
import pytest

from hashinator_gb300 import workloads
from test_bulk_gpu import FILL, _dev, _dt, _host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [4, 8])
def test_requests_far_above_the_round_limit(hx, w):
    import torch
    srv = hx.Server(key_bytes=w, memory_budget=1 << 30, max_maps=2, max_round_requests=3, max_round_keys=1 << 10)
    n = 300_007  # 1172 tiles; the buffers start with room for 8
    m = srv.add_map(20)
    k = workloads.distinct_keys(2 * n, w, 31)
    v = workloads.values(n, w, 31)
    dk, dv = _dev(k), _dev(v)
    out = _dev(np.full(2 * n, FILL, _dt(w)))
    torch.cuda.synchronize()
    kp, vp, op = dk.data_ptr(), dv.data_ptr(), out.data_ptr()
    gone = n // 3
    srv.submit([(m, hx.OP_INSERT, kp, vp, 0, n, 0), (m, hx.OP_ERASE, kp, 0, 0, gone, 1),
                (m, hx.OP_QUERY, kp, 0, op, 2 * n, 2)])
    srv.drain()
    assert [(t, s) for t, _, s in srv.poll()] == [(0, 0), (1, 0), (2, 0)]
    want = np.full(2 * n, FILL, _dt(w))
    want[gone:n] = v[gone:]
    np.testing.assert_array_equal(_host(out, w), want)
    inf = srv.map_info(m)
    assert (inf.fill, inf.tombstone_counter) == (n - gone, gone)
    srv.close()
