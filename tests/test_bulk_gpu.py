"""The slice-by-slice batches against the general path (chosen by a probe
geometry of the caller's own) and against plain numpy: sizes at and around the
rule's lines, ragged sizes, repeated keys, sentinels, pairs and index inserts,
keys that crowd into few buckets (full bins, runs of full buckets across a
slice's or the table's end), tombstones, and a resize. Integer work: the
tolerance is zero."""
import numpy as np
import pytest

from hashinator_gb300 import workloads

pytestmark = pytest.mark.gpu

FILL = 0xA5A5A5A5
SP = {4: 24, 8: 23}  # tables of 128 MiB


def _dt(w):
    return np.uint32 if w == 4 else np.uint64


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32 if a.dtype.itemsize == 4 else np.int64)).cuda()


def _host(t, w):
    return t.cpu().numpy().view(_dt(w))


def _keys_with_homes(home, w, sp, seed):
    """One key per entry of `home`: the inverse of the Fibonacci hash at a random product with those top bits."""
    rng = np.random.default_rng(seed)
    bits = 8 * w
    s = bits - sp
    low = rng.integers(0, 1 << min(s, 62), size=len(home), dtype=np.uint64)
    x = (home.astype(np.uint64) << np.uint64(s)) | low
    mul = {4: 2654435769, 8: 11400714819323198485}[w]
    with np.errstate(over="ignore"):
        x = x * np.uint64(pow(mul, -1, 1 << bits))
    if w == 4:
        x &= np.uint64(0xFFFFFFFF)
    t = s
    while t < bits:
        x ^= x >> np.uint64(t)
        t *= 2
    x = np.unique(x.astype(_dt(w)))
    return rng.permutation(x[x < np.iinfo(_dt(w)).max - 1])


def _asked(n, extra, rng):
    """The numbers of n present and `extra` absent keys, shuffled."""
    return rng.permutation(n + extra)


def _expect(vals, at, w, alive=None):
    """The look-up of keys number `at` where the first len(vals) are in the map (or those of them that are alive)."""
    v = np.concatenate([vals, np.zeros(1, vals.dtype)])
    here = at < len(vals)
    at = np.where(here, at, len(vals))
    if alive is not None:
        here &= np.concatenate([alive, np.zeros(1, bool)])[at]
    return np.where(here, v[at], _dt(w)(FILL))


def _look(m, q, w, general=False):
    """Look-up of q, sentinel-filled; general: by the general path."""
    out = _dev(np.full(len(q), FILL, _dt(w)))
    if general:
        m.set_tuning(group_width=8)
    m.retrieve(_dev(q), out)
    return _host(out, w)


def _check(hx, w, sp, keys, vals, absent, erase_frac=0.4):
    """Insert distinct keys, look present and absent ones up, erase some (twice each), look up again; a second map does
    the same by the general path."""
    rng = np.random.default_rng(len(keys))
    n = len(keys)
    m, g = hx.Hashmap(sp, w), hx.Hashmap(sp, w)
    g.set_tuning(group_width=1)
    for x in (m, g):
        x.insert(_dev(keys), _dev(vals), target_lf=0.0)
    assert m.info().fill == g.info().fill == n
    assert m.peek_status() == hx.STATUS_SUCCESS
    at = _asked(n, len(absent), rng)
    q = np.concatenate([keys, absent])[at]
    want = _expect(vals, at, w)
    np.testing.assert_array_equal(_look(m, q, w), want)
    np.testing.assert_array_equal(_look(g, q, w), want)
    gone = rng.permutation(n)[:int(n * erase_frac)]
    twice = rng.permutation(np.concatenate([keys[gone], keys[gone], absent[:len(absent) // 2]]))
    for x in (m, g):
        x.erase(_dev(twice))
    im, ig = m.info(), g.info()
    assert (im.fill, im.tombstone_counter) == (ig.fill, ig.tombstone_counter) == (n - len(gone), len(gone))
    alive = np.ones(n, bool)
    alive[gone] = False
    np.testing.assert_array_equal(_look(m, q, w), _expect(vals, at, w, alive))
    # back in with new values for every key, over the tombstones where they leave room (inserts never reuse them)
    if n + len(gone) > 0.95 * (1 << sp):
        m.clean_tombstones()
    new = vals[::-1].copy()
    m.insert(_dev(keys), _dev(new), target_lf=0.0)
    assert m.info().fill == n
    want = _expect(new, at, w)
    np.testing.assert_array_equal(_look(m, q, w), want)
    np.testing.assert_array_equal(_look(m, q, w, general=True), want)
    m.close()
    g.close()


def _random(n, w, seed, extra):
    k = workloads.distinct_keys(n + extra, w, seed)
    return k[:n], workloads.values(n, w, seed), k[n:]


@pytest.mark.parametrize("w", [4, 8])
@pytest.mark.parametrize("num,den,ragged", [(1, 4, 0), (1, 4, -1), (1, 2, 13), (3, 4, 1), (9, 10, -7), (15, 16, 5)])
def test_random_keys(hx, w, num, den, ragged):
    n = (num << SP[w]) // den + ragged
    keys, vals, absent = _random(n, w, 11 * num + den + w, n // 3)
    _check(hx, w, SP[w], keys, vals, absent)


@pytest.mark.parametrize("w,sp", [(4, 21), (8, 20), (4, 22)])
def test_small_dense_tables(hx, w, sp):
    n = int(0.92 * (1 << sp)) + 3
    keys, vals, absent = _random(n, w, sp + w, n // 2)
    _check(hx, w, sp, keys, vals, absent)


@pytest.mark.parametrize("w", [4, 8])
@pytest.mark.parametrize("width,per_home", [(1, 40), (300, 2), (2600, 2), (40, 220)])
def test_crowded_homes(hx, w, width, per_home):
    """Crowds of keys around the ends of slices and of the table, on top of evenly spread ones: runs of up to thousands
    of full buckets that cross into the next slice (or wrap), and bins that fill up."""
    sp = SP[w]
    slots, slice_ = 1 << sp, 1 << (12 if w == 4 else 11)
    rng = np.random.default_rng(width + per_home)
    ends = np.array([1, 2, 77, slots // slice_]) * slice_
    crowd = np.concatenate([np.repeat(np.arange(e - width, e), per_home) for e in ends]) % slots
    even = rng.integers(0, slots, size=slots // 2, dtype=np.int64)
    k = _keys_with_homes(np.concatenate([crowd, even]), w, sp, width)
    cut = len(k) * 4 // 5
    keys, absent = k[:cut], k[cut:]
    vals = rng.integers(0, np.iinfo(_dt(w)).max, size=len(keys), dtype=_dt(w))
    _check(hx, w, sp, keys, vals, absent)


@pytest.mark.parametrize("w", [4, 8])
def test_repeated_and_sentinel_keys(hx, w):
    """Every key several times with the same value, one key very often, and the two sentinels in between."""
    n = (1 << SP[w]) // 5
    keys, vals, absent = _random(n, w, 5, n)
    rng = np.random.default_rng(9)
    pick = np.concatenate([np.arange(n), rng.integers(0, n, size=n), np.zeros(1 << 19, np.int64)])
    rng.shuffle(pick)
    k, v = keys[pick], vals[pick]
    top = np.iinfo(_dt(w)).max
    k[::1001], v[::1001] = top, 1
    k[7::1003], v[7::1003] = top - 1, 2
    alive = np.zeros(n, bool)
    alive[pick[(k != top) & (k != top - 1)]] = True
    m = hx.Hashmap(SP[w], w)
    m.insert(_dev(k), _dev(v), target_lf=0.0)
    assert m.info().fill == alive.sum()
    q = np.concatenate([keys, absent, k])
    want = _expect(vals, np.concatenate([np.arange(2 * n), pick]), w, alive)
    want[(q == top) | (q == top - 1)] = FILL
    np.testing.assert_array_equal(_look(m, q, w), want)
    m.erase(_dev(k))
    inf = m.info()
    assert (inf.fill, inf.tombstone_counter) == (0, alive.sum())
    np.testing.assert_array_equal(_look(m, q, w), np.full(len(q), FILL, _dt(w)))
    m.close()


@pytest.mark.parametrize("w", [4, 8])
def test_pairs_index_and_resize(hx, w):
    import torch
    n = (1 << SP[w]) // 2 - 3
    keys, vals, absent = _random(n, w, 21, n // 2)
    m = hx.Hashmap(SP[w], w)
    m.insert_pairs(_dev(np.stack([keys, vals], 1).reshape(-1)), target_lf=0.0)
    assert m.info().fill == n
    at = _asked(n, len(absent), np.random.default_rng(22))
    q = np.concatenate([keys, absent])[at]
    pairs = _dev(np.stack([q, np.full(len(q), FILL, _dt(w))], 1).reshape(-1))
    m.retrieve_pairs(pairs)
    got = _host(pairs, w).reshape(-1, 2)
    np.testing.assert_array_equal(got[:, 0], q)
    want = _expect(vals, at, w)
    np.testing.assert_array_equal(got[:, 1], want)
    m.resize(SP[w] + 1)
    assert m.info().fill == n and m.getSizePower() == SP[w] + 1
    np.testing.assert_array_equal(_look(m, q, w), want)
    m.clear()
    m.insert_index(_dev(keys), target_lf=0.0)
    assert m.info().fill == n
    want = _expect(np.arange(n, dtype=_dt(w)), at, w)
    np.testing.assert_array_equal(_look(m, q, w), want)
    # two look-ups of one map on two streams at once: each has scratch of its own
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    dq = _dev(q)
    outs = [_dev(np.full(len(q), FILL, _dt(w))) for _ in range(4)]
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        m.retrieve(dq, o, stream=(a, b)[i % 2])
    torch.cuda.synchronize()
    for o in outs:
        np.testing.assert_array_equal(_host(o, w), want)
    m.close()


def test_full_table_reports_failure(hx):
    """More keys than buckets: the table fills up, the call reports it, and what is in the table is found."""
    sp = 21
    keys, vals, _ = _random((1 << sp) + 3000, 4, 3, 0)
    m = hx.Hashmap(sp, 4)
    m.insert(_dev(keys[:1 << 20]), _dev(vals[:1 << 20]), target_lf=0.0)
    m.insert(_dev(keys[1 << 20:(1 << 21) - 5000]), _dev(vals[1 << 20:(1 << 21) - 5000]), target_lf=0.0)
    assert m.peek_status() == hx.STATUS_SUCCESS
    m.info()
    m.insert(_dev(keys[(1 << 20):]), _dev(vals[(1 << 20):]), target_lf=0.0)
    assert m.peek_status() == hx.STATUS_FAIL
    assert m.info().fill == 1 << sp
    out = _look(m, keys, 4)
    hit = out == vals
    assert hit.sum() >= (1 << sp) - 8  # (a value may equal the fill by chance)
    assert (out[~hit] == FILL).all()
    m.close()
