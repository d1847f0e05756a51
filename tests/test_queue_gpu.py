"""The automatic insert, look-up and erase kernels (one thread per key, probes
that go on wait in a queue of the warp) where they can go wrong: the smallest
tables, tables that are exactly full, probes that wrap, batches that end in the
middle of a warp, keys repeated within a warp, and more keys than one per
thread; each against the general kernels (a probe geometry of the caller's) and
numpy. Integer work: the tolerance is zero."""
import numpy as np
import pytest

from hashinator_gb300 import workloads
from test_bulk_gpu import FILL, _dev, _dt, _expect, _host, _keys_with_homes

pytestmark = pytest.mark.gpu


def _cycle(hx, w, sp, keys, vals, absent, pairs=False):
    n = len(keys)
    rng = np.random.default_rng(n + sp)
    at = rng.permutation(n + len(absent))
    q = np.concatenate([keys, absent])[at]
    gone = rng.permutation(n)[:(n + 2) // 3]
    alive = np.ones(n, bool)
    alive[gone] = False
    maps = [hx.Hashmap(sp, w), hx.Hashmap(sp, w)]
    maps[1].set_tuning(group_width=2)

    def look(m):
        if pairs:
            p = _dev(np.stack([q, np.full(len(q), FILL, _dt(w))], 1).reshape(-1))
            m.retrieve_pairs(p)
            got = _host(p, w).reshape(-1, 2)
            np.testing.assert_array_equal(got[:, 0], q)
            return got[:, 1]
        out = _dev(np.full(len(q), FILL, _dt(w)))
        m.retrieve(_dev(q), out)
        return _host(out, w)

    for m in maps:
        if pairs:
            m.insert_pairs(_dev(np.stack([keys, vals], 1).reshape(-1)), target_lf=0.0)
        else:
            m.insert(_dev(keys), _dev(vals), target_lf=0.0)
        assert (m.info().fill, m.peek_status()) == (n, hx.STATUS_SUCCESS)
        np.testing.assert_array_equal(look(m), _expect(vals, at, w))
        m.insert(_dev(keys[::-1].copy()), _dev(vals[::-1].copy() + 1), target_lf=0.0)  # every value anew
        assert (m.info().fill, m.peek_status()) == (n, hx.STATUS_SUCCESS)
        np.testing.assert_array_equal(look(m), _expect(vals + 1, at, w))
        m.erase(_dev(np.concatenate([keys[gone], keys[gone[:5]], absent])))
        inf = m.info()
        assert (inf.fill, inf.tombstone_counter) == (n - len(gone), len(gone))
        np.testing.assert_array_equal(look(m), _expect(vals + 1, at, w, alive))
        m.close()


@pytest.mark.parametrize("w", [4, 8])
@pytest.mark.parametrize("sp", [1, 2, 3, 4, 5, 8, 11])
@pytest.mark.parametrize("free", [0, 1, 0.5])
def test_small_and_full_tables(hx, w, sp, free):
    n = (1 << sp) - (free if free >= 1 else int(free * (1 << sp)))
    n = max(int(n), 1)
    k = workloads.distinct_keys(n + 70, w, sp)
    _cycle(hx, w, sp, k[:n], workloads.values(n, w, sp), k[n:], pairs=sp == 4)


@pytest.mark.parametrize("w", [4, 8])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 70001, (1 << 19) + 5])
def test_ragged_batches(hx, w, n):
    sp = int(np.ceil(np.log2(n / 0.78))) + 1 if n < 1000 else int(np.ceil(np.log2(n / 0.9)))
    k = workloads.distinct_keys(2 * n + 9, w, n)
    _cycle(hx, w, max(sp, 2), k[:n], workloads.values(n, w, n), k[n:])


@pytest.mark.parametrize("w", [4, 8])
def test_one_home_and_the_tables_end(hx, w):
    """Hundreds of keys with one home, and a crowd whose probes wrap round the table's end."""
    sp = 13
    home = np.concatenate([np.full(400, 77), np.full(300, (1 << sp) - 1), np.arange((1 << sp) - 500, 1 << sp)])
    k = _keys_with_homes(home, w, sp, 3)
    n = len(k) * 2 // 3
    _cycle(hx, w, sp, k[:n], workloads.values(n, w, 8), k[n:], pairs=True)


@pytest.mark.parametrize("w", [4, 8])
def test_more_keys_than_buckets(hx, w):
    sp = 9
    k = workloads.distinct_keys(700, w, 2)
    v = workloads.values(700, w, 2)
    m = hx.Hashmap(sp, w)
    m.insert(_dev(k), _dev(v), target_lf=0.0)
    assert m.peek_status() == hx.STATUS_FAIL
    assert m.info().fill == 1 << sp
    m.insert(_dev(k[:0]), _dev(v[:0]), target_lf=0.0)  # an empty insert resets the status
    assert m.peek_status() == hx.STATUS_SUCCESS
    m.clear()
    m.insert(_dev(k[:100]), _dev(v[:100]), target_lf=0.0)  # after a clear the status needs no write
    assert m.peek_status() == hx.STATUS_SUCCESS
    m.insert(_dev(k), _dev(v), target_lf=0.0)
    assert m.peek_status() == hx.STATUS_FAIL
    m.insert(_dev(k[:0]), _dev(v[:0]), target_lf=0.0)
    assert m.peek_status() == hx.STATUS_SUCCESS
    m.close()


@pytest.mark.parametrize("w", [4, 8])
def test_keys_repeated_within_a_warp(hx, w):
    n = 5000
    k = workloads.distinct_keys(n, w, 4)
    v = workloads.values(n, w, 4)
    pick = np.concatenate([np.repeat(np.arange(40), 64), np.random.default_rng(1).integers(0, n, 20000)])
    m = hx.Hashmap(13, w)
    m.insert(_dev(k[pick]), _dev(v[pick]), target_lf=0.0)
    assert m.info().fill == len(np.unique(pick))
    out = _dev(np.full(n, FILL, _dt(w)))
    m.retrieve(_dev(k), out)
    here = np.isin(np.arange(n), pick)
    np.testing.assert_array_equal(_host(out, w), np.where(here, v, _dt(w)(FILL)))
    m.close()
