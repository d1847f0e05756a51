"""The serving loop's host code without a GPU (host_runtime.py): what it writes stays in
its buffers, and a round that cannot have the memory it asks for is not lost."""
import pytest

from host_runtime import run_on_host


@pytest.mark.parametrize("requests,round_keys,sp,n", [
    (4096, 1 << 24, 27, 40_000_000),   # the default server, one request above the round's keys
    (64, 1 << 23, 26, 18_900_001),
    (2, 1 << 10, 22, 1_000_003),       # hundreds of times the round's keys
    (1, 1, 10, 700),
])
def test_a_request_above_the_round_limit_stays_in_its_tile_buffers(tmp_path, requests, round_keys, sp, n):
    run_on_host(tmp_path, f"""
srv = hx.Server(key_bytes=8, memory_budget=1 << 40, max_maps=3, max_round_requests={requests}, max_round_keys={round_keys},
                rounds_in_flight=2)
m = srv.add_map({sp})
for i in range(3):
    srv.submit([(m, op, KEYS, KEYS, KEYS, {n}, 10 * i + op) for op in (hx.OP_INSERT, hx.OP_QUERY, hx.OP_ERASE)])
    srv.submit([(m, hx.OP_QUERY, KEYS, 0, KEYS, 5, 10 * i + 3)])
    srv.drain()
assert sorted((t, s) for t, _, s in srv.poll()) == [(10 * i + j, 0) for i in range(3) for j in range(4)]
srv.close()
""")


def test_a_round_whose_tiles_get_no_memory_waits_for_the_next_step(tmp_path):
    run_on_host(tmp_path, """
srv = hx.Server(key_bytes=4, memory_budget=1 << 40, max_maps=3, max_round_requests=4, max_round_keys=1 << 10)
m = srv.add_map(22)
srv.submit([(m, hx.OP_QUERY, KEYS, 0, KEYS, 100_000, 1), (m, hx.OP_QUERY, KEYS, 0, KEYS, 7, 2)])
lib.fake_fail_host(1)
try:
    srv.step()
    raise SystemExit("no error")
except hx.HXError as e:
    assert e.status == hx.HX_ERR_OOM, e.status
assert srv.poll() == []
srv.drain()
assert [(t, s) for t, _, s in srv.poll()] == [(1, 0), (2, 0)]
srv.close()
""")
