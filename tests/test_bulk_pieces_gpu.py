"""Batches of more keys than go slice by slice at once (2^27): look-ups, erases, pairs
and index inserts in two pieces, the second one short and ragged; and an insert of more
keys than the table has buckets, with repeats, in many. Integer work: the tolerance is
zero."""
import pytest

pytestmark = pytest.mark.gpu

FILL = -8
PIECE = 1 << 27


def _mix(i):
    """A bijection of the 32-bit words (as int64 in [0, 2^32))."""
    m = 0xFFFFFFFF
    x = (i ^ (i >> 16)) * 0x85EBCA6B & m
    x = (x ^ (x >> 13)) * 0xC2B2AE35 & m
    return x ^ (x >> 16)


def _keys(lo, hi, w):
    """Distinct keys number lo .. hi - 1, no sentinel among them."""
    import torch
    k = _mix(torch.arange(lo, hi, device="cuda", dtype=torch.int64))
    if w == 8:
        return k * 0x9E3779B1 + 7
    k = torch.where(k >= 1 << 31, k - (1 << 32), k).to(torch.int32)
    assert int((k >= -2).logical_and(k < 0).sum()) == 0
    return k


@pytest.mark.parametrize("w", [4, 8])
def test_look_ups_and_erases_in_two_pieces(hx, w):
    import torch
    n, sp = PIECE + 100_003, 28
    m = hx.Hashmap(sp, w)
    keys = _keys(0, n, w)
    vals = keys ^ 0x5A5A5A5
    m.insert(keys, vals, target_lf=1.0)
    assert m.info().fill == n and m.peek_status() == hx.STATUS_SUCCESS
    out = torch.full_like(vals, FILL)
    m.retrieve(keys, out)
    assert torch.equal(out, vals)
    # the second piece asks for absent keys between present ones
    ask = keys.clone()
    ask[PIECE::2] = _keys(n, n + len(ask[PIECE::2]), w)
    want = vals.clone()
    want[PIECE::2] = FILL
    out.fill_(FILL)
    m.retrieve(ask, out)
    assert torch.equal(out, want)
    pairs = torch.stack([ask, torch.full_like(ask, FILL)], 1).contiguous()
    m.retrieve_pairs(pairs)
    assert torch.equal(pairs[:, 0], ask) and torch.equal(pairs[:, 1], want)
    del pairs
    m.erase(ask)
    left = (n - PIECE + 1) // 2
    inf = m.info()
    assert (inf.fill, inf.tombstone_counter) == (left, n - left)
    out.fill_(FILL)
    m.retrieve(keys, out)
    want.fill_(FILL)
    want[PIECE::2] = vals[PIECE::2]
    assert torch.equal(out, want)
    m.close()


@pytest.mark.parametrize("w", [4, 8])
def test_pairs_and_index_inserts_in_two_pieces(hx, w):
    import torch
    n, sp = PIECE + 77_777, 28
    m = hx.Hashmap(sp, w)
    keys = _keys(0, n, w)
    vals = torch.arange(n, device="cuda").to(keys.dtype)
    m.insert_index(keys, target_lf=1.0)
    out = torch.full_like(vals, FILL)
    m.retrieve(keys, out)
    assert m.info().fill == n and torch.equal(out, vals)
    m.clear()
    m.insert_pairs(torch.stack([keys, ~vals], 1).contiguous(), target_lf=1.0)
    m.retrieve(keys, out)
    assert m.info().fill == n and torch.equal(out, ~vals)
    m.close()


@pytest.mark.parametrize("w", [4, 8])
def test_more_keys_than_buckets_with_repeats(hx, w):
    import torch
    sp = 24
    n = 3 << (sp - 2)
    g = torch.Generator(device="cuda").manual_seed(w)
    distinct = _keys(0, n, w)
    pick = torch.cat([torch.randperm(n, device="cuda", generator=g), torch.randint(0, n, (4 * n + 12345,), device="cuda",
                                                                                  generator=g)])
    pick = pick[torch.randperm(len(pick), device="cuda", generator=g)]
    keys = distinct[pick].contiguous()
    m = hx.Hashmap(sp, w)
    m.insert_pairs(torch.stack([keys, keys ^ 3], 1).contiguous(), target_lf=0.0)
    assert m.info().fill == n and m.peek_status() == hx.STATUS_SUCCESS
    out = torch.full_like(distinct, FILL)
    m.retrieve(distinct, out)
    assert torch.equal(out, distinct ^ 3)
    m.clear()
    m.insert_index(keys, target_lf=0.0)  # each key keeps one of its numbers
    out.fill_(FILL)
    m.retrieve(distinct, out)
    assert m.info().fill == n and torch.equal(keys[out.to(torch.int64)], distinct)
    m.close()
