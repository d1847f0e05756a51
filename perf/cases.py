"""The work this framework is timed on, case by case.

Each case is one pass of a user's program through the public entry points
(`Hashmap`, `tools`, `Batch`, `Server`) on device-resident inputs. Every map
case uses distinct keys from a bijective stream (so each result is known), an
output buffer that starts as a fill value (a missing key leaves its element as
it was), and the default tuning.

Kinds:

* rebuild  one time step that rebuilds a map: clear, insert, look up, erase a
           quarter, clean_tombstones, look up again. Small sizes are the
           per-step calls of a fine-grained program, where launches count.
* build    clear, insert, look up: the bulk load and probe of a large table.
* churn    one step of a long-lived dense map: the keys erased in the step
           before come back, all are looked up, the same share is erased and
           the tombstones are cleaned.
* ingest   a new map of the default size that grows while chunks arrive, then
           one look-up of everything.
* copy_if  stable compaction of an array by a rule, with the count returned.
* scan     exclusive prefix sum of 32-bit words.
* extract  the pairs with an even value, and all keys, of a map in bucket order.
* batch    one round over many per-cell maps (velocity-block ids of a shell in
           a 200^3 grid): insert, look up, erase, clean in one launch, then a
           look-up of the erased keys.
* serve    a burst of insert / look-up / erase requests over resident maps.
"""
import math

import numpy as np
import torch

import hashinator_gb300 as hx

M32 = 0xFFFFFFFF
FILL = -8  # what the output of an absent key keeps


def listed():
    return [
        # A small map rebuilt every step: six calls whose launches outweigh their work.
        {"name": "rebuild_u32_small", "kind": "rebuild", "width": 4, "sp": 10, "n": 499, "hit": 0.5},
        # An ordinary 64-bit map, ragged size; the table (4 MiB) stays in L2.
        {"name": "rebuild_u64_ordinary", "kind": "rebuild", "width": 8, "sp": 18, "n": 100003, "hit": 0.5},
        # The single-map test configuration: 2^20 keys at load factor 0.5.
        {"name": "rebuild_u32_2p20", "kind": "rebuild", "width": 4, "sp": 21, "n": 1 << 20, "hit": 0.5},
        # The benchmark's headline step: 2^26 keys into 2^27 buckets, as many look-ups, half of them present.
        {"name": "build_u32_2p26", "kind": "build", "width": 4, "sp": 27, "n": 1 << 26, "hit": 0.5},
        # The large 64-bit table of the load-factor sweep, three quarters full.
        {"name": "build_u64_lf075", "kind": "build", "width": 8, "sp": 27, "n": 3 << 25, "hit": 0.5},
        # The densest table of the sweep over one step of its life: 30 % of the keys leave and come back.
        {"name": "churn_u32_lf090", "kind": "churn", "width": 4, "sp": 27, "n": 120795955, "hit": 0.5},
        # Keys arriving in chunks of a ragged size at a map that starts small and grows.
        {"name": "ingest_u32_growth", "kind": "ingest", "width": 4, "n": 20000003, "chunks": 6, "hit": 0.5},
        # The streaming benchmark: 2^28 words, the rule x % 100 < 50.
        {"name": "copy_if_u32_2p28", "kind": "copy_if", "elem": 4, "n": 1 << 28, "s": 50},
        # The scan of the streaming benchmark at a size that is no multiple of any tile.
        {"name": "scan_u32_ragged", "kind": "scan", "n": (1 << 28) - 57},
        # extractPattern and extractAllKeys over a half-full table of 2^27 buckets.
        {"name": "extract_u32_2p27", "kind": "extract", "width": 4, "sp": 27, "n": 1 << 26},
        # The batched configuration: 4096 per-cell maps of 2^6 to 2^16 keys.
        {"name": "batch_4096_maps", "kind": "batch", "maps": 4096, "log_hi": 16.0},
        # A burst at the serving loop: 64-bit maps of 2^8 to 2^17 keys, requests of 1 to 2^14 keys.
        {"name": "serve_u64_256maps", "kind": "serve", "maps": 256, "requests": 2048, "log_req": 14.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rebuild", "rebuild", "rebuild", "build", "build", "churn", "churn", "ingest", "copy_if", "copy_if",
                       "scan", "extract", "batch", "serve"])
    if kind in ("rebuild", "build", "churn"):
        lo, hi = {"rebuild": (5, 22), "build": (22, 27), "churn": (10, 27)}[kind]
        sp = rng.randint(lo, hi)
        lf = rng.uniform(0.3, 0.5 if kind == "rebuild" else 0.9)
        return {"kind": kind, "width": rng.choice([4, 8]), "sp": sp, "n": max(4, int(lf * (1 << sp))),
                "hit": round(rng.uniform(0.1, 0.9), 2)}
    if kind == "ingest":
        return {"kind": kind, "width": rng.choice([4, 8]), "n": _log_int(rng, 5000, 20000000), "chunks": rng.randint(2, 8),
                "hit": round(rng.uniform(0.1, 0.9), 2)}
    if kind == "copy_if":
        elem = rng.choice([4, 4, 8, 16])
        return {"kind": kind, "elem": elem, "n": _log_int(rng, 1000, (1 << 30) // elem), "s": rng.choice([1, 10, 50, 90, 99])}
    if kind == "scan":
        return {"kind": kind, "n": _log_int(rng, 1000, 1 << 28)}
    if kind == "extract":
        sp = rng.randint(10, 26)
        return {"kind": kind, "width": rng.choice([4, 8]), "sp": sp, "n": int(rng.uniform(0.2, 0.8) * (1 << sp))}
    if kind == "batch":
        return {"kind": kind, "maps": _log_int(rng, 16, 4096), "log_hi": round(rng.uniform(8.0, 16.0), 2)}
    return {"kind": "serve", "maps": _log_int(rng, 8, 256), "requests": _log_int(rng, 64, 2048),
            "log_req": round(rng.uniform(6.0, 14.0), 2)}


# ---- inputs -----------------------------------------------------------------


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + salt)


def _i32(x):
    """int64 values in [0, 2^32) as the same 32 bits."""
    return torch.where(x >= 1 << 31, x - (1 << 32), x).to(torch.int32)


def _mix32(i, salt):
    x = i ^ (salt & M32)
    x = x ^ (x >> 16)
    x = (x * 0x85EBCA6B) & M32
    x = x ^ (x >> 13)
    x = (x * 0xC2B2AE35) & M32
    return x ^ (x >> 16)


def _signed(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def _shr(x, s):
    return (x >> s) & ((1 << (64 - s)) - 1)


def _mix64(i, salt):
    z = i ^ _signed(salt * 0x9E3779B97F4A7C15)
    z = (z ^ _shr(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ _shr(z, 31)


def _stream(n, width, seed, offset=0):
    """n distinct keys from stream positions [offset, ...), none of them a sentinel."""
    pos = torch.arange(offset, offset + n + 2, device="cuda", dtype=torch.int64)
    k = _i32(_mix32(pos, seed * 7919 + 13)) if width == 4 else _mix64(pos, seed * 7919 + 13)
    return k[(k != -1) & (k != -2)][:n].contiguous()


def _dtype(width):
    return torch.int32 if width == 4 else torch.int64


def _values(n, width, g):
    if width == 4:
        return torch.randint(-(1 << 31), (1 << 31) - 1, (n,), device="cuda", dtype=torch.int32, generator=g)
    return torch.randint(-(1 << 62), (1 << 62) - 1, (n,), device="cuda", dtype=torch.int64, generator=g)


def _map_inputs(case, seed):
    """Keys, values, look-ups (a shuffled mix of present and absent keys), and for each look-up the index of the key it
    asks for (-1: absent); and the indices of the keys that the step erases."""
    width, n = case["width"], case["n"]
    g = _gen(seed)
    keys = _stream(n, width, seed)
    vals = _values(n, width, g)
    n_hit = int(round(n * case["hit"]))
    at = torch.full((n,), -1, device="cuda", dtype=torch.int64)
    at[:n_hit] = torch.randperm(n, device="cuda", generator=g)[:n_hit]
    at = at[torch.randperm(n, device="cuda", generator=g)]
    q = torch.empty_like(keys)
    hit = at >= 0
    q[hit] = keys[at[hit]]
    q[~hit] = _stream(n - n_hit, width, seed, offset=n + 64)
    share = 0.3 if case["kind"] == "churn" else 0.25
    gone = torch.randperm(n, device="cuda", generator=g)[:int(n * share)]
    return keys, vals, q, at, gone


def _looked_up(vals, at, gone=None):
    if gone is not None:
        alive = torch.ones(len(vals), device="cuda", dtype=torch.bool)
        alive[gone] = False
        at = torch.where((at >= 0) & alive[at.clamp(min=0)], at, torch.full_like(at, -1))
    return torch.where(at >= 0, vals[at.clamp(min=0)], torch.full_like(vals[:1], FILL))


def _home_keys(sp, width, n, seed):
    """n distinct keys with distinct home buckets, spread over a table of 2^sp buckets, and those buckets in order:
    each key is the inverse of the Fibonacci hash at a random product whose top bits are the bucket. A table of such
    keys has one layout, whatever order they are inserted in."""
    g = _gen(seed, 1)
    home = torch.sort(torch.randperm(1 << sp, device="cuda", generator=g)[:n]).values
    if width == 4:
        s = 32 - sp
        p = (home << s) | torch.randint(0, 1 << s, (n,), device="cuda", dtype=torch.int64, generator=g)
        x = (p * pow(2654435769, -1, 1 << 32)) & M32
        while s < 32:
            x = x ^ (x >> s)
            s *= 2
        k = _i32(x)
    else:
        s = 64 - sp
        low = torch.randint(0, 1 << min(s, 62), (n,), device="cuda", dtype=torch.int64, generator=g)
        x = ((home << s) | low) * _signed(pow(11400714819323198485, -1, 1 << 64))
        while s < 64:
            x = x ^ _shr(x, s)
            s *= 2
        k = x
    return k[(k != -1) & (k != -2)].contiguous()


def _elements(case, seed):
    """copy_if's input as rows of 1 (u32) or 2 (key, value) words; keys of pairs are never sentinels here."""
    n, elem = case["n"], case["elem"]
    g = _gen(seed)
    if elem == 4:
        return _values(n, 4, g)
    return _values(2 * n, elem // 2, g)


def _copy_rule(case):
    if case["elem"] == 4:
        return hx.Pred.mod_lt(100, case["s"])
    # pairs: the value's low bits against a bound give the same share of selected elements
    return hx.Pred.value_even() if case["s"] == 50 else hx.Pred(hx.PRED_MOD_LT, hx.FIELD_VALUE, 100, case["s"])


def _copy_selected(case, x):
    """The rule in 64-bit arithmetic, one truth value an element."""
    if case["elem"] == 4:
        return (x.to(torch.int64) & M32) % 100 < case["s"]
    v = x.view(-1, 2)[:, 1]
    k = x.view(-1, 2)[:, 0]
    if case["s"] == 50:
        return (v & 1 == 0) & (k != -1) & (k != -2)
    if case["elem"] == 8:
        return (v.to(torch.int64) & M32) % 100 < case["s"]
    # an unsigned 64-bit value mod 100 from its signed reading (2^64 mod 100 = 16)
    return (torch.remainder(v, 100) + torch.where(v < 0, 16, 0)) % 100 < case["s"]


_SHELL = {}


def _shell():
    """Offsets of the cells between 30 and 60 cells from the centre, as one id each in a 200^3 grid."""
    if "ids" not in _SHELL:
        ax = torch.arange(-60, 61, device="cuda", dtype=torch.int64)
        x, y, z = torch.meshgrid(ax, ax, ax, indexing="ij")
        d2 = x * x + y * y + z * z
        _SHELL["ids"] = (x + 200 * (y + 200 * z))[(d2 >= 900) & (d2 <= 3600)].contiguous()
    return _SHELL["ids"]


_PRIMES = (1000003, 1299709, 2750159, 4256233, 15485863, 32452843)  # above every modulus below, so coprime to it


def _segments(sizes):
    """(segment, index within it) of every element of a concatenation of segments."""
    seg = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), sizes)
    start = torch.cumsum(sizes, 0) - sizes
    return seg, torch.arange(len(seg), device="cuda") - start[seg], start


def _offsets(sizes):
    o = np.zeros(len(sizes) + 1, np.uint64)
    o[1:] = np.cumsum(sizes.cpu().numpy())
    return o


def _sizes(count, lo, hi):
    """`count` sizes spread log-uniformly over [2^lo, 2^hi], in a scattered order: the same ones for every seed."""
    return np.rint(2.0 ** (lo + (hi - lo) * ((np.arange(count) + 0.5) * 0.6180339887498949 % 1.0))).astype(np.int64)


def _batch_inputs(case, seed):
    """Per map n_i = 2^U distinct velocity-block ids, n_i look-ups (70 % present), a tenth erased. Random draws within a
    map are affine permutations j -> (a j + b) mod m with a prime a above m."""
    g, maps = _gen(seed), case["maps"]
    n = torch.from_numpy(_sizes(maps, 6.0, case["log_hi"])).cuda()
    primes = torch.tensor(_PRIMES, device="cuda")

    def affine():
        return (primes[torch.randint(0, len(_PRIMES), (maps,), device="cuda", generator=g)],
                torch.randint(0, 1 << 30, (maps,), device="cuda", generator=g))

    shell = _shell()
    centre = torch.randint(60, 140, (maps, 3), device="cuda", generator=g)
    centre = centre[:, 0] + 200 * (centre[:, 1] + 200 * centre[:, 2])
    n_hit = torch.round(n * 0.7).to(torch.int64)
    n_gone = torch.round(n * 0.1).to(torch.int64)
    a, b = affine()

    def ids(seg, j):
        return (shell[(a[seg] * j + b[seg]) % len(shell)] + centre[seg]).to(torch.int32)

    seg, j, start = _segments(n)
    keys, vals = ids(seg, j), _values(len(seg), 4, g)
    c, d = affine()
    e, f = affine()
    where = (c[seg] * j + d[seg]) % n[seg]            # the look-up's number in its map, shuffled
    number = (e[seg] * where + f[seg]) % n[seg]       # a permutation of the map's keys: the first n_hit are asked for
    present = where < n_hit[seg]
    q = ids(seg, torch.where(present, number, n[seg] + where))  # ids past the n inserted ones are absent
    at = torch.where(present, start[seg] + number, torch.full_like(j, -1))
    u, w = affine()
    gseg, gj, _ = _segments(n_gone)
    gone = keys[start[gseg] + (u[gseg] * gj + w[gseg]) % n[gseg]].contiguous()
    sp = torch.ceil(torch.log2(n.to(torch.float64) * 2)).to(torch.int32).cpu().numpy()
    return {"sp": sp, "keys": keys, "vals": vals, "q": q.contiguous(), "at": at, "gone": gone,
            "off": _offsets(n), "gone_off": _offsets(n_gone)}


def _serve_inputs(case, seed):
    """Resident maps and one burst of requests on them. Half of a map's keys are reserved for insert / erase pairs (an
    insert request brings some of them and a later erase request takes the same ones), the other half are looked up, so
    every look-up's answer is known; 80 % of the looked-up keys are present. About 15 % of the requests are inserts and
    as many erases."""
    shape = np.random.default_rng(case["requests"])  # sizes, maps and order: the same for every seed
    rng = np.random.default_rng(seed)                # which keys
    maps, n_req = case["maps"], case["requests"]
    n0 = _sizes(maps, 8.0, 17.0)
    sp = np.maximum(np.ceil(np.log2(n0 / 0.5)), 2).astype(np.int64)
    start = np.cumsum(n0) - n0
    used = np.zeros(maps, np.int64)
    slots = shape.permutation(n_req)
    reqs, i = [], 0
    while i < n_req:
        m = int(shape.integers(maps))
        k = int(max(1, round(2.0 ** shape.uniform(0.0, case["log_req"]))))
        if i + 1 < n_req and shape.random() < 0.18:
            k = min(k, int(n0[m] // 2 - used[m]))
            if k > 0:
                pos = np.arange(used[m], used[m] + k)
                used[m] += k
                first, last = sorted((int(slots[i]), int(slots[i + 1])))
                reqs += [(first, m, hx.OP_INSERT, pos), (last, m, hx.OP_ERASE, pos)]
                i += 2
                continue
            k = 1
        there = rng.random(k) < 0.8
        pos = np.where(there, rng.integers(n0[m] // 2, n0[m], size=k), n0[m] + (1 << 24) + rng.integers(1 << 24, size=k))
        reqs.append((int(slots[i]), m, hx.OP_QUERY, pos))
        i += 1
    reqs.sort(key=lambda r: r[0])
    length = np.array([len(r[3]) for r in reqs], np.int64)
    off = np.cumsum(length) - length
    which = np.concatenate([r[3] for r in reqs])
    of = np.repeat([r[1] for r in reqs], length)
    asks = np.repeat([r[2] == hx.OP_QUERY for r in reqs], length)
    at = np.where(which < n0[of], start[of] + which, -1)
    salt = seed * 7919 + 13
    init = np.concatenate([np.arange(k) + (m << 40) for m, k in enumerate(n0)])
    keys = _mix64(torch.from_numpy(init).cuda(), salt)
    req_keys = _mix64(torch.from_numpy(which + (of << 40)).cuda(), salt)
    vals = _values(len(keys), 8, _gen(seed))
    at = torch.from_numpy(at).cuda()
    asks = torch.from_numpy(asks).cuda()
    return {"sp": sp, "n0": n0, "start": start, "keys": keys, "vals": vals, "reqs": reqs, "off": off, "req_keys": req_keys,
            "req_vals": vals[at.clamp(min=0)].contiguous(), "at": at, "asks": asks}


# ---- the interface ------------------------------------------------------------


def prepare(case, seed):
    kind, s = case["kind"], {"kind": case["kind"]}
    if kind in ("rebuild", "build", "churn"):
        keys, vals, q, at, gone = _map_inputs(case, seed)
        s |= {"keys": keys, "vals": vals, "q": q, "gone": keys[gone].contiguous(), "gone_vals": vals[gone].contiguous(),
              "out": torch.full_like(q, FILL), "out2": torch.full_like(q, FILL)}
        s["map"] = hx.Hashmap(case["sp"], case["width"])
        if kind == "churn":
            m = s["map"]
            m.insert(keys, vals, target_lf=1.0)
            m.erase(s["gone"])
            m.clean_tombstones()
            m.info()
    elif kind == "ingest":
        keys, vals, q, at, gone = _map_inputs(case, seed)
        step = -(-len(keys) // case["chunks"])
        s |= {"width": case["width"], "chunks": [(keys[a:a + step], vals[a:a + step]) for a in range(0, len(keys), step)],
              "q": q, "out": torch.full_like(q, FILL)}
    elif kind == "copy_if":
        x = _elements(case, seed)
        s |= {"x": x, "out": torch.full_like(x, 0), "rule": _copy_rule(case), "elem": case["elem"]}
    elif kind == "scan":
        x = torch.randint(0, 16, (case["n"],), device="cuda", dtype=torch.int32, generator=_gen(seed))
        s |= {"x": x, "out": torch.zeros_like(x)}
    elif kind == "extract":
        keys = _home_keys(case["sp"], case["width"], case["n"], seed)
        vals = _values(len(keys), case["width"], _gen(seed))
        m = hx.Hashmap(case["sp"], case["width"])
        order = torch.randperm(len(keys), device="cuda", generator=_gen(seed, 2))
        m.insert(keys[order].contiguous(), vals[order].contiguous(), target_lf=1.0)
        s |= {"map": m, "pairs": torch.zeros(2 * len(keys), device="cuda", dtype=_dtype(case["width"])),
              "keys": torch.zeros_like(keys)}
    elif kind == "batch":
        w = _batch_inputs(case, seed)
        b = hx.Batch(w["sp"])
        out = torch.full_like(w["q"], FILL)
        out2 = torch.full_like(w["gone"], FILL)
        s |= {"w": w, "batch": b, "out": out, "out2": out2,
              "round": b.plan(w["keys"], w["vals"], w["off"], w["q"], out, w["off"], w["gone"], w["gone_off"], clean=True),
              "after": b.plan(query_keys=w["gone"], query_out=out2, query_offsets=w["gone_off"])}
    else:
        w = _serve_inputs(case, seed)
        srv = hx.Server(key_bytes=8, memory_budget=16 << 30, max_load_factor=0.8, max_maps=case["maps"])
        ids = [srv.add_map(int(p)) for p in w["sp"]]
        k0, v0 = w["keys"].data_ptr(), w["vals"].data_ptr()
        srv.submit([(ids[m], hx.OP_INSERT, k0 + 8 * int(a), v0 + 8 * int(a), 0, int(n), m)
                    for m, (a, n) in enumerate(zip(w["start"], w["n0"]))])
        srv.drain()
        srv.poll()
        out = torch.full_like(w["req_keys"], FILL)
        k, v, o = w["req_keys"].data_ptr(), w["req_vals"].data_ptr(), out.data_ptr()
        s |= {"w": w, "srv": srv, "out": out,
              "reqs": srv.requests([(ids[m], op, k + 8 * int(a), v + 8 * int(a), o + 8 * int(a), len(pos), i)
                                    for i, ((_, m, op, pos), a) in enumerate(zip(w["reqs"], w["off"]))])}
    torch.cuda.synchronize()  # the inputs are ready before the server's own stream reads them
    return s


def run(s):
    kind = s["kind"]
    if kind == "rebuild":
        m = s["map"]
        m.clear()
        m.insert(s["keys"], s["vals"])
        m.retrieve(s["q"], s["out"])
        m.erase(s["gone"])
        m.clean_tombstones()
        m.retrieve(s["q"], s["out2"])
        return s["out"], s["out2"]
    if kind == "build":
        m = s["map"]
        m.clear()
        m.insert(s["keys"], s["vals"], target_lf=1.0)
        m.retrieve(s["q"], s["out"])
        return s["out"]
    if kind == "churn":
        m = s["map"]
        m.insert(s["gone"], s["gone_vals"], target_lf=1.0)
        m.retrieve(s["q"], s["out"])
        m.erase(s["gone"])
        m.clean_tombstones()
        return s["out"], m.info().fill
    if kind == "ingest":
        m = hx.Hashmap(key_bytes=s["width"])
        for k, v in s["chunks"]:
            m.insert(k, v)
        m.retrieve(s["q"], s["out"])
        m.close()
        return s["out"]
    if kind == "copy_if":
        return hx.tools.copy_if(s["x"], s["out"], s["rule"], elem_bytes=s["elem"]), s["out"]
    if kind == "scan":
        hx.tools.split_prefix_scan(s["x"], s["out"])
        return s["out"]
    if kind == "extract":
        m = s["map"]
        return (m.extract_pattern(hx.Pred.value_even(), s["pairs"]), s["pairs"], m.extract_all_keys(s["keys"]), s["keys"])
    if kind == "batch":
        s["batch"].clear()
        s["round"].run_graph()
        s["after"].run_graph()
        return s["out"], s["out2"]
    srv = s["srv"]
    srv.submit(s["reqs"])
    srv.drain()
    srv.poll(capacity=len(s["reqs"]))
    return s["out"]


def work(case):
    """Bytes of one pass: every input array read once, every output element written once, and one pass over the bucket
    array for each call that has to see or set all of it (clear, clean_tombstones, extraction). A look-up, an insert or
    an erase of a large table cannot do without the bucket it changes or reads: pair bytes each, in either direction
    that it uses, but no more than the array itself."""
    kind = case["kind"]
    if kind in ("rebuild", "build", "churn", "ingest"):
        w, n = case["width"], case["n"]
        if kind == "ingest":
            sp = math.ceil(math.log2(n / 0.5))
        else:
            sp = case["sp"]
        table = 2 * w << sp

        def touch(k, both):
            return min(2 * w * k, table) * (2 if both else 1)

        look = 2 * w * n + touch(n, False)
        ins = 2 * w * n + touch(n, True)
        if kind == "rebuild":
            gone = int(0.25 * n)
            return {"bytes": table + ins + 2 * look + w * gone + touch(gone, True) + table}
        if kind == "build":
            return {"bytes": table + ins + look}
        if kind == "churn":
            gone = int(0.3 * n)
            return {"bytes": 2 * w * gone + touch(gone, True) + look + w * gone + touch(gone, True) + table}
        return {"bytes": ins + look + table}
    if kind == "copy_if":
        return {"bytes": case["n"] * case["elem"] * (1 + case["s"] / 100)}
    if kind == "scan":
        return {"bytes": 8 * case["n"]}
    if kind == "extract":
        return {"bytes": 2 * (2 * case["width"] << case["sp"]) + 2 * case["width"] * case["n"]}
    if kind == "batch":
        mean = (2.0 ** case["log_hi"] - 64) / ((case["log_hi"] - 6.0) * math.log(2.0))
        n = case["maps"] * mean
        table = 8 * 2.7 * n
        return {"bytes": 2 * table + 8 * n * 2 + 8 * 0.7 * n * 2 + 4 * 0.1 * n * 2}
    mean = (2.0 ** case["log_req"] - 1) / (case["log_req"] * math.log(2.0))
    return {"bytes": case["requests"] * mean * (8 + 16 + 8)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("rebuild", "build", "churn", "ingest"):
        _, vals, _, at, gone = _map_inputs(case, seed)
        out = _looked_up(vals, at)
        if kind == "rebuild":
            return out, _looked_up(vals, at, gone)
        if kind == "churn":
            return out, len(vals) - len(gone)
        return out
    if kind == "copy_if":
        x = _elements(case, seed)
        sel = _copy_selected(case, x)
        got = (x if case["elem"] == 4 else x.view(-1, 2))[sel].reshape(-1)
        out = torch.zeros_like(x)
        out[:len(got)] = got
        return int(sel.sum()), out
    if kind == "scan":
        x = torch.randint(0, 16, (case["n"],), device="cuda", dtype=torch.int32, generator=_gen(seed))
        c = torch.cumsum(x.to(torch.int64), 0) - x
        return _i32(c & M32)
    if kind == "extract":
        keys = _home_keys(case["sp"], case["width"], case["n"], seed)
        vals = _values(len(keys), case["width"], _gen(seed))
        even = vals & 1 == 0
        got = torch.stack((keys[even], vals[even]), 1).reshape(-1)
        pairs = torch.zeros(2 * len(keys), device="cuda", dtype=keys.dtype)
        pairs[:len(got)] = got
        return int(even.sum()), pairs, len(keys), keys
    if kind == "batch":
        w = _batch_inputs(case, seed)
        return _looked_up(w["vals"], w["at"]), torch.full_like(w["gone"], FILL)
    w = _serve_inputs(case, seed)
    at = torch.where(w["asks"], w["at"], torch.full_like(w["at"], -1))
    return _looked_up(w["vals"], at)
