"""The memory that libhx holds after a large table is gone is bounded, and other
allocations of the process can have it."""
import pytest

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_freed_tables_go_back_to_the_device(hx):
    import gc
    import torch
    gc.collect()  # maps of earlier tests
    torch.cuda.empty_cache()
    hx.Hashmap(10, 4).close()
    start = _free()  # the pool may still hold the 1 GiB that it keeps without a map
    small = hx.Hashmap(10, 4)
    big = hx.Hashmap(20, 8)
    big.resize(30)  # 16 GiB
    assert start - _free() >= 15 * GIB
    big.resize(22)
    assert start - _free() <= 5 * GIB + (1 << 27)
    big.resize(30)
    big.close()
    assert start - _free() <= 5 * GIB + (1 << 27)
    small.close()
    assert start - _free() <= 1 * GIB + (1 << 27)
