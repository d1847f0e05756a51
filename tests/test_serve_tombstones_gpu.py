"""A map whose keys come and go is rehashed once its probes run long through the
tombstones they leave: after many rounds that insert and erase the same keys,
look-ups are still exact and the longest probe stays short. Integer work: the
tolerance is zero."""
import numpy as np
import pytest

from hashinator_gb300 import workloads
from test_bulk_gpu import FILL, _dev, _dt, _host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [4, 8])
def test_long_probes_through_tombstones_are_cut(hx, w):
    import torch
    srv = hx.Server(key_bytes=w, memory_budget=1 << 28, max_load_factor=0.8, max_maps=2)
    sp, n, rounds = 12, 900, 200
    ids = [srv.add_map(sp), srv.add_map(sp)]
    k = workloads.distinct_keys(n + 300, w, 6)
    v = workloads.values(n + 300, w, 6)
    dk, dv = _dev(k), _dev(v)
    out = _dev(np.full(2 * (n + 300), FILL, _dt(w)))
    torch.cuda.synchronize()
    size = dk.element_size()
    kp, vp, op = dk.data_ptr(), dv.data_ptr(), out.data_ptr()
    come = 7  # the keys n .. n + 7 come and go in the first map
    srv.submit([(i, hx.OP_INSERT, kp, vp, 0, n, 0) for i in ids])
    srv.drain()
    for _ in range(rounds):
        srv.submit([(ids[0], hx.OP_INSERT, kp + n * size, vp + n * size, 0, come, 1),
                    (ids[0], hx.OP_ERASE, kp + n * size, 0, 0, come, 2)])
        srv.drain()
    assert {s for _, _, s in srv.poll()} == {0}
    srv.submit([(ids[0], hx.OP_QUERY, kp, 0, op, n + 300, 3),
                (ids[1], hx.OP_QUERY, kp, 0, op + (n + 300) * size, n + 300, 4)])
    srv.drain()
    got = _host(out, w)
    want = np.where(np.arange(n + 300) < n, v, _dt(w)(FILL))
    np.testing.assert_array_equal(got, np.concatenate([want, want]))
    inf = [srv.map_info(i) for i in ids]
    assert [i.fill for i in inf] == [n, n] and [i.size_power for i in inf] == [sp, sp]
    # each round lengthens the probe to one home by one bucket: without rehashes the bound would pass `rounds`
    assert inf[0].max_probe < rounds // 2 and srv.stats()["growths"] >= 1
    assert inf[1].tombstone_counter == 0
    srv.close()
