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


# Two maps of 2^12 u64 buckets. snap() plays a round's metadata: the longest probe of map 0
# grows tenfold while its tombstones do, which asks for a rehash at its size.
TANGLED = """
class DInfo(ctypes.Structure):
    _fields_ = [("fill", ctypes.c_uint64), ("tombstones", ctypes.c_uint64), ("max_probe", ctypes.c_uint32)]
    _pad_ = 72
def server(budget):
    s = hx.Server(key_bytes=8, memory_budget=budget, max_load_factor=0.8, max_maps=5)
    assert [s.add_map(12), s.add_map(12)] == [0, 1]
    ctypes.memset(lib.fake_find(5 * 72), 0, 5 * 72)
    return s
def snap(s, probe, tombs, fill=500):
    d = DInfo.from_address(lib.fake_find(5 * 72))
    d.fill, d.tombstones, d.max_probe = fill, tombs, probe
    s.submit([(1, hx.OP_QUERY, KEYS, 0, KEYS, 3, 0)])
    s.drain()
    s.poll()
def go(s, reqs):
    s.submit([(m, op, KEYS, KEYS, KEYS, n, i) for i, (m, op, n) in enumerate(reqs)])
    s.drain()
    return [st for _, _, st in sorted(s.poll())]
def at(s):
    return [s.bucket_data(i) for i in range(2)]
INSERT, QUERY, ERASE = hx.OP_INSERT, hx.OP_QUERY, hx.OP_ERASE
"""


def test_tombstones_are_dropped_before_an_insert_and_only_then(tmp_path):
    run_on_host(tmp_path, TANGLED + """
s = server(1 << 30)
snap(s, 20, 0)
snap(s, 200, 100)
before = at(s)
# look-ups and erases leave a table where it is: a caller may hold its address
assert go(s, [(0, QUERY, 5), (0, ERASE, 5)]) == [0, 0]
assert at(s) == before and s.stats()["growths"] == 0
assert go(s, [(0, QUERY, 5), (0, INSERT, 5)]) == [0, 0]
assert at(s)[0] != before[0] and at(s)[0][1] == 1 << 12 and at(s)[1] == before[1] and s.stats()["growths"] == 1
""")


def test_a_probe_bound_that_grows_with_the_keys_asks_for_no_rehash(tmp_path):
    run_on_host(tmp_path, TANGLED + """
s = server(1 << 30)
snap(s, 20, 0, 500)
snap(s, 150, 10, 3000)   # long, but ten tombstones cannot be the reason
snap(s, 180, 60, 3000)
before = at(s)
assert go(s, [(0, INSERT, 5)]) == [0]
assert at(s) == before and s.stats()["growths"] == 0
""")


def test_a_rehash_for_speed_takes_no_memory_that_is_not_there(tmp_path):
    run_on_host(tmp_path, TANGLED + """
s = server((2 << 16) + (1 << 15))  # room for the two tables and half of another
snap(s, 20, 0)
snap(s, 200, 100)
before = at(s)
assert go(s, [(0, INSERT, 5)]) == [0]
assert at(s) == before and s.stats()["growths"] == 0

s = server(1 << 30)
snap(s, 20, 0)
snap(s, 200, 100)
before = at(s)
lib.fake_fail_pool_from(1)
assert go(s, [(0, INSERT, 5), (1, QUERY, 5)]) == [0, 0]
assert at(s) == before and s.stats()["growths"] == 0
lib.fake_fail_pool_from(0)
snap(s, 500, 300)
assert go(s, [(0, INSERT, 5)]) == [0]  # it is tried again later
assert at(s)[0] != before[0] and s.stats()["growths"] == 1
""")


def test_an_insert_whose_table_cannot_be_had_is_rejected_and_the_others_run(tmp_path):
    run_on_host(tmp_path, TANGLED + """
s = server(1 << 30)
before, used = at(s), s.memory()[0]
lib.fake_fail_pool_from(1 << 20)  # a table of 2^13 buckets can be had, one of 2^16 cannot
assert go(s, [(0, INSERT, 4000), (1, INSERT, 50000), (1, QUERY, 5), (1, INSERT, 50)]) == [0, hx.HX_ERR_OOM, 0, 0]
assert at(s)[0][1] == 1 << 13 and at(s)[1] == before[1]
st = s.stats()
assert (st["growths"], st["rejected"]) == (1, 1) and s.memory()[0] == used + (1 << 16)
""")
