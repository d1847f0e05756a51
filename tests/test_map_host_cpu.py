"""A map's host-side bookkeeping without a GPU (host_runtime.py): what a replay of a
captured call changes on the device is not taken for known."""
from host_runtime import run_on_host

INFO = """
class DInfo(ctypes.Structure):
    _fields_ = [("fill", ctypes.c_uint64), ("tombstones", ctypes.c_uint64), ("max_probe", ctypes.c_uint32),
                ("err", ctypes.c_int32)]
def dinfo():
    return DInfo.from_address(lib.fake_find(72))
FAIL = hx.STATUS_FAIL
"""


def test_status_after_a_replay_between_clear_and_insert(tmp_path):
    run_on_host(tmp_path, INFO + """
m = hx.Hashmap(10, 4)
d = dinfo()
for captured in (False, True):
    if captured:
        lib.fake_capture(1)
        m.insert(KEYS, KEYS, n=100, target_lf=0.0)
        lib.fake_capture(0)
    m.clear()
    d.err = 0            # what the clear kernel leaves
    if captured:
        d.err = FAIL     # what a replay that fills the table leaves
    m.insert(KEYS, KEYS, n=10, target_lf=0.0)
    assert d.err == 0, (captured, d.err)
""")


def test_scratch_of_captured_calls(tmp_path):
    run_on_host(tmp_path, INFO + """
lib.fake_live.argtypes = [ctypes.c_int]
pred, count = hx.Pred.value_even().c(), 1 << 12
mem = ctypes.c_uint64()
def extract(m):  # with the count left on the device
    assert lib.hx_extract_pattern(m._m, ctypes.byref(pred), KEYS, 100, ctypes.addressof(mem), None, None) == 0
m = hx.Hashmap(20, 4)
lib.fake_capture(1)
extract(m)
m.insert(KEYS, KEYS, n=1 << 18, target_lf=0.0)
m.clean_tombstones()
lib.fake_capture(0)
assert lib.fake_live(1) == 0  # the map keeps nothing that belongs to the graph
extract(m)                    # takes a buffer of the map's own
lib.fake_capture(1)
extract(m)                    # replays use that buffer
lib.fake_capture(0)
held = lib.fake_live(0)
m.clean_tombstones()          # takes a larger one: the graph's lives on
assert lib.fake_live(0) == held + 1 and lib.fake_live(1) == 0
m.close()
assert lib.fake_live(0) == 0
""")


def test_growth_after_a_replay(tmp_path):
    run_on_host(tmp_path, INFO + """
def size_power(m):
    return m.bucket_data()[1].bit_length() - 1
m = hx.Hashmap(10, 4)
lib.fake_capture(1)
m.insert(KEYS, KEYS, n=400, target_lf=0.5)  # in a capture the bound decides: nothing is read back
lib.fake_capture(0)
m.clear()
dinfo().fill = 900  # what a replay leaves
m.insert(KEYS, KEYS, n=200, target_lf=0.5)
assert size_power(m) == 12
""")
