"""clean_tombstones on tables of one slice and of several (a slice is 4096 u32
or 2048 u64 buckets), from two buckets up: the counters, the number of keys
taken out, the probe bound and the table's layout against the bucket array read
back before and after, with evenly spread keys and with crowds whose runs cross
the ends of slices and of the table. Integer work: the tolerance is zero."""
import numpy as np
import pytest

from gpu_util import bucket_array
from test_bulk_gpu import _dev, _dt, _host, _keys_with_homes

pytestmark = pytest.mark.gpu

FILL = 0xA5A5A5A5


def _home(k, w, sp):
    bits = 8 * w
    k = k.astype(np.uint64)
    k ^= k >> np.uint64(bits - sp)
    with np.errstate(over="ignore"):
        p = k * np.uint64({4: 2654435769, 8: 11400714819323198485}[w])
    if w == 4:
        p &= np.uint64(0xFFFFFFFF)
    return (p >> np.uint64(bits - sp)).astype(np.int64)


def _layout(b, w, sp):
    """Keys, their distances from home and whether each can be reached (no EMPTY bucket from its home to it)."""
    top = np.iinfo(_dt(w)).max
    n = 1 << sp
    at = np.flatnonzero(b[:, 0] < top - 1)
    dist = (at - _home(b[at, 0], w, sp)) % n
    empty = np.concatenate([b[:, 0] == top] * 2)
    before = np.concatenate([[0], np.cumsum(empty)])
    reach = before[at + n] - before[at + n - dist] == 0
    return b[at, 0], dist, reach


def _run(hx, w, sp, keys, vals, erase_frac, seed):
    rng = np.random.default_rng(seed)
    m = hx.Hashmap(sp, w)
    if len(keys):
        m.insert(_dev(keys), _dev(vals), target_lf=0.0)
    assert m.info().fill == len(keys)
    m.clean_tombstones()  # no tombstones: nothing happens
    assert m.info().last_clean_moved == 0
    gone = rng.permutation(len(keys))[:int(np.ceil(len(keys) * erase_frac))]
    if len(gone):
        m.erase(_dev(keys[gone]))
    b = bucket_array(m, w)
    _, dist, _ = _layout(b, w, sp)
    m.clean_tombstones()
    inf = m.info()
    assert (inf.fill, inf.tombstone_counter) == (len(keys) - len(gone), 0)
    assert m.peek_status() == hx.STATUS_SUCCESS
    if len(gone):
        assert inf.last_clean_moved == (dist > 0).sum()
    a = bucket_array(m, w)
    top = np.iinfo(_dt(w)).max
    assert not (a[:, 0] == top - 1).any()
    assert (a[a[:, 0] == top, 1] == 0).all()
    k, dist, reach = _layout(a, w, sp)
    alive = np.ones(len(keys), bool)
    alive[gone] = False
    np.testing.assert_array_equal(np.sort(k), np.sort(keys[alive]))
    assert reach.all()
    if len(gone):
        assert inf.max_probe == (dist.max() + 1 if len(dist) else 0)
    out = _dev(np.full(len(keys), FILL, _dt(w)))
    if len(keys):
        m.retrieve(_dev(keys), out)
        np.testing.assert_array_equal(_host(out, w), np.where(alive, vals, _dt(w)(FILL)))
    m.close()


@pytest.mark.parametrize("w", [4, 8])
@pytest.mark.parametrize("sp", [1, 2, 3, 4, 5, 6, 10, 11, 12, 13, 16])
@pytest.mark.parametrize("lf,erase", [(0.5, 0.3), (0.9, 0.5), (1.0, 0.01), (0.7, 1.0)])
def test_even_keys(hx, w, sp, lf, erase):
    from hashinator_gb300 import workloads
    n = max(1, int(lf * (1 << sp)))
    _run(hx, w, sp, workloads.distinct_keys(n, w, sp + 7), workloads.values(n, w, sp), erase, sp)


@pytest.mark.parametrize("w", [4, 8])
@pytest.mark.parametrize("sp", [12, 14, 17])
@pytest.mark.parametrize("width,per_home", [(1, 30), (60, 12), (900, 2)])
def test_runs_across_slices(hx, w, sp, width, per_home):
    slots, slice_ = 1 << sp, 1 << (12 if w == 4 else 11)
    rng = np.random.default_rng(width + sp)
    ends = np.arange(1, slots // slice_ + 1) * slice_
    crowd = np.concatenate([np.repeat(np.arange(e - width, e), per_home) for e in ends]) % slots
    even = rng.integers(0, slots, size=slots // 6, dtype=np.int64)
    k = _keys_with_homes(np.concatenate([crowd, even]), w, sp, width)[:int(0.97 * slots)]
    for erase in (0.02, 0.6):
        _run(hx, w, sp, k, rng.integers(0, np.iinfo(_dt(w)).max, size=len(k), dtype=_dt(w)), erase, sp)
