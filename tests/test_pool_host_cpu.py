"""How much freed device memory libhx's pool holds, and that it gives it back when an
allocation needs it (host code against a stand-in runtime, host_runtime.py)."""
from host_runtime import run_on_host

GIB = "GIB = 1 << 30\n"


def test_pool_keeps_a_bounded_amount(tmp_path):
    run_on_host(tmp_path, GIB + """
small = hx.Hashmap(10, 4)
big = hx.Hashmap(20, 8)
big.resize(30)  # 16 GiB
assert 16 * GIB <= lib.fake_pool_held() <= 21 * GIB
big.resize(22)
assert lib.fake_pool_held() <= 5 * GIB + (1 << 26), "after the large table is freed"
big.resize(30)
big.close()
assert lib.fake_pool_held() <= 5 * GIB, "after its map is destroyed"
small.close()
assert lib.fake_pool_held() <= 1 * GIB, "after the last map is destroyed"
b = hx.Batch([10, 12])
b.close()
assert lib.fake_pool_held() <= 1 * GIB
""")


def test_pool_gives_way_to_other_allocations(tmp_path):
    run_on_host(tmp_path, GIB + """
lib.fake_capacity(18 * GIB)
def held():  # 4 GiB in the pool, none of them in use
    m = hx.Hashmap(20, 8)
    m.resize(28)
    m.close()
    assert lib.fake_pool_held() >= 4 * GIB
keep = hx.Hashmap(10, 4)
held()
m = hx.Hashmap(30, 8)      # 16 GiB of 18
m.close()
held()
b = hx.Batch([30, 10], key_bytes=8)
b.close()
held()
s = hx.Server(key_bytes=8, memory_budget=40 * GIB, max_maps=2)
assert s.add_map(30) == 0 and s.try_add_map(28) is None
s.close()
""")
