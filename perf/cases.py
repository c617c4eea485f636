"""Workloads of the compression-aware query path, called as a user's program
calls them: columns compressed once and kept in a device arena, then operator
calls whose scratch and results live in the same arena until it is reset for
the next query.

Every case is a dict with an ``op`` and its sizes; ``prepare`` makes the raw
values with torch from the seed, compresses them into the state's arena and
returns what a program keeps between queries, ``run`` is one query.  Values
are random but result sizes are the case's own: hits are spread evenly (one
at a random place in every 1/keep rows), every group occurs, a column of runs
has a fixed number of runs.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

import engine_b200 as ms

FORMATS = {"uncompr": ms.uncompr_f, "dynamic": ms.dynamic_vbp_f, "delta": ms.delta_f, "for": ms.for_f, "rle": ms.rle_f}
FOR_BASE = 1 << 40  # for_f columns: a large common offset (timestamps, surrogate keys)
ZIPF_KEYS = 1000


def listed():
    return [
        # the reference's example query (select -> project -> agg_sum, one
        # operator call each) on a column of a few thousand rows: a lookup in
        # a small table, where launches and host work are all there is
        dict(name="query_small", op="query", n=5003, x="dynamic", xbits=10, y="dynamic", ybits=20, keep=0.5),
        # the same query as one fused call over a large table (an analytical
        # scan; results stay on the device)
        dict(name="fused_scan_large", op="fused", n=1 << 28, x="dynamic", xbits=10, y="dynamic", ybits=20, keep=0.5,
             sync=False),
        # ingest: a column arrives uncompressed and is stored as dynamic_vbp
        dict(name="compress_dynamic", op="compress", n=(1 << 27) + 777, fmt="dynamic", dist="uniform", bits=20),
        # export: a sorted key column kept as deltas is read back uncompressed
        dict(name="decompress_delta", op="decompress", n=(1 << 27) + 333, fmt="delta", dist="sorted", bits=0),
        # a column with runs (a denormalised dimension attribute) stored as
        # rle and read back
        dict(name="rle_roundtrip", op="roundtrip", n=(1 << 26) + 41, fmt="rle", dist="runs", bits=20),
        # filter on one column with compressed positions, projection of
        # another through them, the result recompressed
        dict(name="select_project", op="select_project", n=(1 << 26) + 1029, x="for", xbits=16, y="dynamic", ybits=20,
             keep=0.1, pos="delta", out="dynamic"),
        # a dimension filter on a fact table: semi join of the foreign key
        # with the filtered dimension's keys, intersected with another
        # operator's position list
        dict(name="semi_join_intersect", op="semi_join", n=(1 << 26) + 515, keys=1 << 20, wide=False, keep=0.1,
             fk="dynamic", out="delta"),
        # a key/foreign-key join with both position lists
        dict(name="natural_join", op="natural_join", n=(1 << 25) + 9, keys=1 << 20, wide=False, keep=0.5, fk="dynamic",
             out="uncompr"),
        # group by a skewed key, then sum a measure per group
        dict(name="group_sum", op="group", n=(1 << 25) + 2051, key="dynamic", keys=ZIPF_KEYS, skew=1.1, bits=16),
        # the star query as one fused call over the fact table
        dict(name="star_query", op="star", n=1 << 27, keys=1 << 20, keep=0.1, groups=ZIPF_KEYS),
        # a scan of many columns of very different lengths and formats at
        # once (the plan is built once and replayed)
        dict(name="batch_columns", op="batch", cols=256, lo=10, hi=22),
        # format choice per block by the learned selector, compression into
        # the blockwise container and a scan of it
        dict(name="learned_selector", op="selector", blocks=1 << 15),
    ]


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    def size(lo, hi):
        n = int(2.0 ** rng.uniform(lo, hi))
        return n if rng.random() < 0.25 else n | 1

    op = rng.choice(["query", "fused", "compress", "decompress", "roundtrip", "select_project", "semi_join",
                     "natural_join", "group", "star", "batch", "selector"])
    block = ["uncompr", "static", "dynamic", "for"]
    if op == "query":
        return dict(op=op, n=size(10, 20), x=rng.choice(block), xbits=rng.randint(4, 24), y=rng.choice(block),
                    ybits=rng.randint(4, 40), keep=rng.choice([0.01, 0.1, 0.5, 0.9]))
    if op == "fused":
        return dict(op=op, n=size(12, 27), x=rng.choice(block[1:]), xbits=rng.randint(4, 32), y=rng.choice(block[1:]),
                    ybits=rng.randint(4, 40), keep=rng.choice([0.01, 0.1, 0.5, 0.9]), sync=rng.random() < 0.5)
    if op in ("compress", "decompress", "roundtrip"):
        fmt = rng.choice(["static", "dynamic", "delta", "for"] if op != "roundtrip" else ["rle", "rle", "delta", "for"])
        dist = {"static": "uniform", "dynamic": "uniform", "delta": "sorted", "for": "offset", "rle": "runs"}[fmt]
        if op == "decompress" and fmt in ("dynamic", "delta", "for") and rng.random() < 0.3:
            dist = rng.choice(["zipf", "mixed"])
        return dict(op=op, n=size(12, 26), fmt=fmt, dist=dist, bits=rng.randint(1, 48))
    if op == "select_project":
        return dict(op=op, n=size(12, 25.5), x=rng.choice(block), xbits=rng.randint(4, 24), y=rng.choice(block),
                    ybits=rng.randint(4, 40), keep=rng.choice([0.01, 0.1, 0.5]),
                    pos=rng.choice(["uncompr", "delta", "dynamic", "for"]), out=rng.choice(["uncompr", "dynamic", "for"]))
    if op in ("semi_join", "natural_join"):
        return dict(op=op, n=size(12, 24.5), keys=size(8, 20), wide=rng.random() < 0.3,
                    keep=rng.choice([0.01, 0.1, 0.5]), fk=rng.choice(block),
                    out=rng.choice(["uncompr", "delta", "dynamic"]))
    if op == "group":
        n = size(12, 24)
        return dict(op=op, n=n, key=rng.choice(block), keys=min(rng.choice([8, 100, ZIPF_KEYS, 20000]), n // 4),
                    skew=rng.choice([0.0, 1.1]), bits=rng.randint(8, 32))
    if op == "star":
        n = size(14, 26.5)
        return dict(op=op, n=n, keys=size(10, 20), keep=rng.choice([0.05, 0.1, 0.5]),
                    groups=ZIPF_KEYS if n >= 1 << 26 else 100 if n >= 1 << 22 else 8 if n >= 1 << 18 else 1)
    if op == "batch":
        return dict(op=op, cols=rng.choice([16, 48, 128]), lo=10, hi=rng.choice([16, 20]))
    return dict(op=op, blocks=size(6, 14.5))


# ---------------------------------------------------------------------------
# raw values (torch, from the seed alone)
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _uniform(g, bits, n):
    return torch.randint(0, 1 << min(bits, 62), (n,), dtype=torch.int64, device="cuda", generator=g)


def _zipf(g, s, keys, n):
    w = torch.arange(1, keys + 1, dtype=torch.float64, device="cuda") ** -s
    cdf = torch.cumsum(w / w.sum(), 0)
    u = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    return torch.searchsorted(cdf, u).clamp_(max=keys - 1)


def _sorted(g, n):
    """Ascending keys, gaps 1 + Geom of mean 4, a larger one every 256 rows."""
    u = torch.rand(n, dtype=torch.float32, device="cuda", generator=g).clamp_(min=1e-7)
    gaps = 1 + (torch.log(u) / np.log(0.75)).to(torch.int64)
    gaps[::256] += 300
    return torch.cumsum(gaps, 0)


def _runs(g, bits, n, mean=32):
    """max(1, n / mean) runs of geometric lengths, neighbours different."""
    head = torch.rand(n, device="cuda", generator=g) < 1.0 / mean
    head[0] = True
    want = max(1, n // mean)
    for _ in range(64):  # to the exact number of runs
        extra = int(head.sum().item()) - want
        if not extra:
            break
        at = torch.nonzero(head if extra > 0 else ~head).flatten()
        at = at[at > 0]
        pick = torch.unique((torch.arange(abs(extra), device="cuda") * at.numel()) // abs(extra))
        head[at[pick]] = extra < 0
    run = torch.cumsum(head.to(torch.int64), 0) - 1
    return (_uniform(g, bits, want) * 2 + torch.arange(want, device="cuda") % 2)[run]


def _spread(g, n, keep):
    """A bool mask over n rows: one row at a random place in every 1/keep
    (all but one where keep > 1/2)."""
    q = round(1 / min(keep, 1 - keep))
    m = torch.zeros(n, dtype=torch.bool, device="cuda")
    k = n // q
    m[torch.arange(k, device="cuda") * q + torch.randint(0, q, (k,), device="cuda", generator=g)] = True
    return ~m if keep > 0.5 else m


def _mixed(g, n):
    """Segments of 64 Ki values cycling through families of values."""
    seg = 1 << 16
    parts = []
    for i, at in enumerate(range(0, n, seg)):
        m = min(seg, n - at)
        k = i % 4
        if k == 0:
            parts.append(_uniform(g, 1 + (i * 7) % 40, m))
        elif k == 1:
            parts.append(_sorted(g, m) + (1 << 20))
        elif k == 2:
            parts.append(_runs(g, 20, m))
        else:
            parts.append(_zipf(g, 1.2, 1 << 16, m))
    return torch.cat(parts)


def _column(g, fmt, bits, n):
    """Values for a column of the given format: for_f ones far from zero."""
    v = _uniform(g, bits, n)
    return v + FOR_BASE if fmt == "for" else v


def _cut(fmt, bits, keep):
    """The filter's constant: a `keep` share of its column lies below it."""
    return max(1, int(keep * (1 << bits))) + (FOR_BASE if fmt == "for" else 0)


def _filter_column(g, fmt, bits, n, keep):
    c = _cut("", bits, keep)
    v = torch.where(_spread(g, n, keep), torch.randint(0, c, (n,), dtype=torch.int64, device="cuda", generator=g),
                    torch.randint(c, 1 << bits, (n,), dtype=torch.int64, device="cuda", generator=g))
    return v + FOR_BASE if fmt == "for" else v


def _dist(g, case):
    n, b = case["n"], case["bits"]
    d = case["dist"]
    if d == "uniform":
        return _uniform(g, b, n)
    if d == "offset":
        return _uniform(g, b, n) + FOR_BASE
    if d == "sorted":
        return _sorted(g, n)
    if d == "runs":
        return _runs(g, min(b, 40), n)
    if d == "zipf":
        return _zipf(g, 1.2, 1 << 20, n)
    return _mixed(g, n)


def _dim(g, case):
    """The filtered dimension's keys, a sorted `keep` share of [0, keys) spread
    over 2^40 where `wide`, and the keys that the filter dropped."""
    m = _spread(g, case["keys"], case["keep"])
    k = torch.arange(case["keys"], dtype=torch.int64, device="cuda") * _stride(case)
    return k[m], k[~m]


def _pick(g, values, n):
    return values[torch.randint(0, values.numel(), (n,), device="cuda", generator=g)]


def _stride(case):
    return ((1 << 40) // case["keys"]) if case["wide"] else 1


def _raw(case, seed):
    """The case's uncompressed columns as int64 CUDA tensors."""
    g = _gen(seed)
    op = case["op"]
    if op in ("query", "fused", "select_project"):
        return {"x": _filter_column(g, case["x"], case["xbits"], case["n"], case["keep"]),
                "y": _column(g, case["y"], case["ybits"], case["n"])}
    if op in ("compress", "decompress", "roundtrip"):
        return {"v": _dist(g, case)}
    n = case.get("n", 0)
    if op in ("semi_join", "natural_join"):
        kept, dropped = _dim(g, case)
        hit = _spread(g, n, case["keep"])
        r = {"l": kept, "fk": torch.where(hit, _pick(g, kept, n), _pick(g, dropped, n))}
        if op == "semi_join":
            # another operator's positions: as many rows, every tenth among the hits
            rows, others = torch.nonzero(hit).flatten(), torch.nonzero(~hit).flatten()
            p = others[torch.arange(rows.numel(), device="cuda") * (others.numel() // rows.numel())]
            p[::10] = rows[::10]
            r["p"] = torch.sort(p).values
        return r
    if op == "group":
        k = (_zipf(g, case["skew"], case["keys"], n) if case["skew"] else
             torch.randint(0, case["keys"], (n,), dtype=torch.int64, device="cuda", generator=g))
        at = torch.arange(case["keys"], device="cuda") * (n // case["keys"])
        k[at + torch.randint(0, n // case["keys"], (case["keys"],), device="cuda", generator=g)] = \
            torch.randperm(case["keys"], device="cuda", generator=g)
        return {"k": k + FOR_BASE if case["key"] == "for" else k, "m": _uniform(g, case["bits"], n)}
    if op == "star":
        return {"fk": torch.randint(0, case["keys"], (n,), dtype=torch.int64, device="cuda", generator=g),
                "filter": _uniform(g, 12, n), "gkey": _zipf(g, 1.1, case["groups"], n),
                "measure": _uniform(g, 16, n), "l": _dim(g, dict(case, wide=False))[0]}
    if op == "batch":
        out = {}
        for i, (n, kind, bits) in enumerate(_batch_plan(case)):
            v = (_uniform(g, bits, n) if kind in ("static", "dynamic") else _sorted(g, n) if kind == "delta" else
                 _uniform(g, 16, n) + FOR_BASE if kind == "for" else _runs(g, 20, n))
            out[i] = v
        return out
    return {"v": _mixed(g, case["blocks"] * 2048)}


def _batch_plan(case):
    rng = np.random.default_rng(case["cols"] * 1000 + case["hi"])
    lens = np.floor(2.0 ** rng.uniform(case["lo"], case["hi"], case["cols"])).astype(int)
    kinds = rng.integers(0, 5, case["cols"])
    bits = rng.integers(4, 33, case["cols"])
    names = ("static", "dynamic", "delta", "for", "rle")
    return [(int(n), names[int(k)], int(b)) for n, k, b in zip(lens, kinds, bits)]


def _batch_consts(case, raw):
    return [int(torch.kthvalue(raw[i], raw[i].numel() // 2 + 1).values.item()) for i in range(case["cols"])]


# ---------------------------------------------------------------------------
# device columns
# ---------------------------------------------------------------------------
class _Bytes:
    def __init__(self, arena, ptr, nbytes):
        self.arena = arena  # keeps the memory alive while a tensor uses it
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3}


class Home:
    """The program's device arena: its columns below `mark`, each query's
    scratch and results above it; `new_query` frees the last query's."""

    def __init__(self, nbytes):
        nbytes = (int(nbytes) + 4095) // 4096 * 4096
        self.arena = ms.Arena(nbytes)
        self.base = self.arena.alloc(256)
        self.bytes = torch.as_tensor(_Bytes(self.arena, self.base, nbytes), device="cuda")
        self.mark = 0

    def keep(self):
        self.mark = self.arena.used()

    def new_query(self):
        self.arena.reset()
        self.arena.alloc(self.mark)

    def at(self, ptr, nbytes):
        return self.bytes[ptr - self.base: ptr - self.base + nbytes]

    def words(self, ptr, n):
        return self.at(ptr, 8 * n).view(torch.int64)

    def out(self, col):
        """A result column: values where it is uncompressed, else its
        compressed part and its uncompressed rest (the bytes between the two
        are padding), and its sizes."""
        n, used, compr = col.meta()
        if col.desc.format == ms.UNCOMPR:
            return self.words(col.desc.data, n)
        rest = ms.rest_offset(col.format, compr) if used > compr else used
        return [self.at(col.desc.data, compr), self.at(col.desc.data + rest, used - rest), n, used, compr]


def _format(name, bits):
    return ms.static_vbp_f(max(1, bits)) if name == "static" else FORMATS[name]


def _uncompressed(t):
    n = t.numel()
    return ms.MsCol(format=ms.UNCOMPR, count_values=n, size_used_byte=8 * n, size_alloc_byte=8 * n, data=t.data_ptr())


def _compressed(raws):
    """Every (values, format) compressed into one arena of its own."""
    scratch = ms.Arena((sum(24 * v.numel() for v, _ in raws) + (64 << 20) + 4095) // 4096 * 4096)
    cols = [ms.morph(ms.Column(_uncompressed(v), scratch), f) for v, f in raws]
    return cols, scratch


def _home(raws, room):
    """A Home holding every (values, format) in storage of its own size, and
    `room` bytes for queries."""
    cols, scratch = _compressed(raws)
    need = sum(c.get_size_used_byte() + 9 * c.desc.n_index + 16 * (c.desc.n_index // 2) + 4096 for c in cols)
    home = Home(need + room + (64 << 20))
    kept = [c.compact(home.arena) for c in cols]
    torch.cuda.synchronize()
    scratch.close()
    home.keep()
    return home, kept


def prepare(case, seed):
    op = case["op"]
    raw = _raw(case, seed)
    s = {"case": case}
    if op in ("query", "fused", "select_project"):
        s["home"], (s["x"], s["y"]) = _home([(raw["x"], _format(case["x"], case["xbits"])),
                                             (raw["y"], _format(case["y"], case["ybits"]))],
                                            (4 << 20) if op == "fused" else 48 * case["n"])
        s["c"] = _cut(case["x"], case["xbits"], case["keep"])
        if op == "fused":
            s["sum"], s["count"], s["err"] = (s["home"].arena.alloc(8) for _ in range(3))
            s["home"].words(s["err"], 1).zero_()
            s["home"].keep()
    elif op in ("compress", "roundtrip"):
        s["fmt"] = _format(case["fmt"], case["bits"])
        s["home"], (s["v"],) = _home([(raw["v"], ms.uncompr_f)], 48 * case["n"])
    elif op == "decompress":
        s["home"], (s["v"],) = _home([(raw["v"], _format(case["fmt"], case["bits"]))], 24 * case["n"])
    elif op in ("semi_join", "natural_join"):
        kb = 40 if case["wide"] else (case["keys"] - 1).bit_length()
        cols = [(raw["l"], ms.delta_f), (raw["fk"], _format(case["fk"], kb))]
        if op == "semi_join":
            cols.append((raw["p"], ms.delta_f))
        s["home"], kept = _home(cols, 64 * case["n"] + 64 * case["keys"])
        s.update(zip(("l", "fk", "p"), kept))
    elif op == "group":
        kb = (case["keys"] - 1).bit_length()
        s["home"], (s["k"], s["m"]) = _home([(raw["k"], _format(case["key"], kb)), (raw["m"], ms.dynamic_vbp_f)],
                                            128 * case["n"] + (64 << 20))
    elif op == "star":
        names = ("filter", "fk", "gkey", "measure", "l")
        s["home"], kept = _home([(raw[k], ms.delta_f if k == "l" else ms.dynamic_vbp_f) for k in names], 512 << 20)
        s.update(zip(names, kept))
    elif op == "batch":
        plan = _batch_plan(case)
        s["home"], cols = _home([(raw[i], _format(k, b)) for i, (_, k, b) in enumerate(plan)], 512 << 20)
        s["batch"] = ms.Batch(cols, _batch_consts(case, raw), ms.less, s["home"].arena)
        s["home"].keep()
    else:
        import engine_b200.selector as S
        # a selector trained on blocks of the same kind of data
        train = _raw(dict(case, blocks=2048), seed + 1)["v"]
        n = case["blocks"]
        home = s["home"] = Home(80 * n * 2048 + (256 << 20))
        d = train.data_ptr()
        _, sizes = S.analyze(home.arena, d, 2048)
        s["mlp"] = S.Mlp(seed=1, max_batch=1024)
        s["mlp"].train(home.arena, S.features(home.arena, d, 2048), sizes, 2048, steps=200, batch=1024)
        torch.cuda.synchronize()
        home.arena.reset()
        home.arena.alloc(256)
        s["v"] = home.arena.alloc(8 * n * 2048)
        home.words(s["v"], n * 2048).copy_(raw["v"])
        home.keep()
        torch.cuda.synchronize()
    return s


def run(s):
    case, home = s["case"], s["home"]
    op = case["op"]
    if op == "fused":
        if case["sync"]:
            home.new_query()
            return list(ms.select_project_sum(s["x"], ms.less, s["c"], s["y"]))
        stream = torch.cuda.current_stream().cuda_stream
        ms._check(ms.lib().ms_gpu_select_project_sum_async(C.byref(s["x"].desc), ms.less, s["c"], C.byref(s["y"].desc),
                                                           s["sum"], s["count"], s["err"], stream), "fused scan")
        return [home.words(s["sum"], 1), home.words(s["count"], 1)]
    if op == "batch":
        counts, sums = s["batch"].run(graph=True)
        return [counts, sums]
    home.new_query()
    if op == "query":
        pos = ms.select(ms.less, s["x"], s["c"])
        vals = ms.project(s["y"], pos)
        return [home.out(pos), home.out(vals), ms.agg_sum(vals)]
    if op == "select_project":
        pos = ms.select(ms.less, s["x"], s["c"], FORMATS[case["pos"]])
        return [home.out(pos), home.out(ms.project(s["y"], pos, FORMATS[case["out"]]))]
    if op == "compress":
        return [home.out(ms.morph(s["v"], s["fmt"]))]
    if op == "decompress":
        return [home.out(ms.morph(s["v"], ms.uncompr_f))]
    if op == "roundtrip":
        c = ms.morph(s["v"], s["fmt"])
        return [home.out(c), home.out(ms.morph(c, ms.uncompr_f))]
    if op == "semi_join":
        p2 = ms.semi_join(s["l"], s["fk"], FORMATS[case["out"]])
        return [home.out(p2), home.out(ms.intersect_sorted(s["p"], p2, FORMATS[case["out"]]))]
    if op == "natural_join":
        f = FORMATS[case["out"]]
        return [home.out(c) for c in ms.natural_join(s["l"], s["fk"], f, f)]
    if op == "group":
        gr, ext = ms.group(s["k"])
        return [home.out(gr), home.out(ext), home.out(ms.agg_sum_grouped(gr, s["m"], ext.get_count_values()))]
    if op == "star":
        return list(ms.query3(s["filter"], ms.less, 400, s["fk"], s["l"], s["gkey"], s["measure"]))
    import engine_b200.selector as S
    a, d, n = home.arena, s["v"], case["blocks"]
    feats = S.features(a, d, n)
    choice, _, _ = s["mlp"].choose(a, feats, n, float(np.log2(1.02)))
    S.resolve(d, n, choice)
    stats, _ = S.analyze(a, d, n)
    box = S.Container(a, d, n, stats, choice)
    total, count, _ = box.select_sum(ms.less, 1 << 20)
    return [home.at(feats, 4 * S.NF * n).view(torch.float32), home.at(choice, n), home.words(box.offsets, n),
            home.at(box.codes, n), home.at(box.psz, 4 * n), box.nbytes, total, count]


# ---------------------------------------------------------------------------
# the least bytes of a pass: each input read once, each output written once
# ---------------------------------------------------------------------------
def _cbytes(fmt, bits, n):
    return {"uncompr": 8 * n, "static": bits * n / 8, "dynamic": bits * n / 8 + n / 512,
            "for": bits * n / 8 + n / 1024 * 72, "delta": 7 * n / 8 + n / 16, "rle": 16 * n / 32}[fmt]


def work(case):
    op, n = case["op"], case.get("n", 0)
    if op in ("query", "fused", "select_project"):
        b = _cbytes(case["x"], case["xbits"], n) + _cbytes(case["y"], case["ybits"], n)
        hits = case["keep"] * n
        if op == "query":
            b += 16 * hits
        if op == "select_project":
            b += _cbytes(case["pos"], 26, hits) + _cbytes(case["out"], case["ybits"], hits)
    elif op in ("compress", "decompress", "roundtrip"):
        bits = {"zipf": 20, "mixed": 20, "runs": 20, "sorted": 40}.get(case["dist"], case["bits"])
        b = 8 * n + _cbytes(case["fmt"], bits, n)
        if op == "roundtrip":
            b *= 2
    elif op in ("semi_join", "natural_join"):
        kb = 40 if case["wide"] else (case["keys"] - 1).bit_length()
        hits = case["keep"] * n
        b = _cbytes("delta", 0, case["keep"] * case["keys"]) + _cbytes(case["fk"], kb, n)
        if op == "semi_join":
            b += _cbytes("delta", 0, hits) + _cbytes(case["out"], 26, hits) + _cbytes(case["out"], 26, 0.1 * hits)
        else:
            b += 2 * _cbytes(case["out"], 26, hits)
    elif op == "group":
        b = _cbytes(case["key"], (case["keys"] - 1).bit_length(), n) + _cbytes("dynamic", case["bits"], n) + 8 * n
    elif op == "star":
        b = _cbytes("dynamic", (case["keys"] - 1).bit_length() + 12 + case["groups"].bit_length() + 16, n)
    elif op == "batch":
        b = sum(_cbytes(k, 16 if k == "for" else bits, m) for m, k, bits in _batch_plan(case))
    else:
        b = 8 * 2048 * case["blocks"] * 1.3
    return {"bytes": int(b), "flops": 0}


# ---------------------------------------------------------------------------
# the results in plain 64-bit torch
# ---------------------------------------------------------------------------
def _features(v):
    """The learned selector's block statistics, computed in 64 bits: bit-width
    histograms, extremes, delta signs and run heads over four runs of 64
    values at 0, 512, 1024 and 1536 of every block."""
    x = v.view(-1, 4, 512)[:, :, :64]
    d = x[:, :, 8:] - x[:, :, :-8]

    def width(t):
        w = torch.ones(t.shape, dtype=torch.int64, device=t.device)
        for k in range(1, 64):
            w += ((t >> k) & ((1 << (64 - k)) - 1) if k else t) != 0
        return w

    wv, wd = width(x), width(d)
    nd = float(d[0].numel())
    f = []
    for w, cnt in ((wv, 256.0), (wd, nd)):
        for k in range(8):
            f.append((((w - 1) >> 3) == k).sum((1, 2)).double() / cnt)
    hi, lo = x.amax((1, 2)), x.amin((1, 2))
    heads = (x[:, :, 1:] != x[:, :, :-1]).sum((1, 2)).double()
    f += [wv.amax((1, 2)).double() / 64, wv.amin((1, 2)).double() / 64, width(hi - lo).double() / 64,
          wd.amax((1, 2)).double() / 64, (d < 0).sum((1, 2)).double() / nd, heads / 252,
          (d == 0).sum((1, 2)).double() / nd, wv.sum((1, 2)).double() / (256 * 64)]
    f += [wv[:, c].amax(1).double() / 64 for c in range(4)] + [wd[:, c].amax(1).double() / 64 for c in range(4)]
    return torch.stack(f, 1).flatten()


def _groups(keys):
    """(group id per row, first row of every group), ids in order of first
    occurrence."""
    u, inv = torch.unique(keys, return_inverse=True)
    n = keys.numel()
    first = torch.full((u.numel(),), n, dtype=torch.int64, device=keys.device)
    first.scatter_reduce_(0, inv, torch.arange(n, device=keys.device), reduce="amin")
    order = torch.argsort(first)
    rank = torch.empty_like(order)
    rank[order] = torch.arange(order.numel(), device=keys.device)
    return rank[inv], first[order]


def _opaque(fmt, values):
    """A result column: its values where it is uncompressed, else nothing to
    compute (its bytes are the format's)."""
    return values if fmt == "uncompr" else [None] * 5


def exact(case, seed):
    op = case["op"]
    if op == "compress" or (op == "select_project" and "uncompr" not in (case["pos"], case["out"])) or \
            (op in ("semi_join", "natural_join") and case["out"] != "uncompr"):
        return None  # the results are bytes of a format
    raw = _raw(case, seed)
    if op in ("query", "fused", "select_project"):
        pos = torch.nonzero(raw["x"] < _cut(case["x"], case["xbits"], case["keep"])).flatten()
        vals = raw["y"][pos]
        if op == "query":
            return [pos, vals, int(vals.sum().item())]
        if op == "fused":
            s, k = int(vals.sum().item()), pos.numel()
            return [s, k] if case["sync"] else [torch.tensor([s], device="cuda"), torch.tensor([k], device="cuda")]
        return [_opaque(case["pos"], pos), _opaque(case["out"], vals)]
    if op == "decompress":
        return [raw["v"]]
    if op == "roundtrip":
        return [[None] * 5, raw["v"]]
    if op in ("semi_join", "natural_join"):
        l, fk = raw["l"], raw["fk"]
        at = torch.searchsorted(l, fk).clamp_(max=max(l.numel() - 1, 0))
        hit = (l[at] == fk) if l.numel() else torch.zeros_like(fk, dtype=torch.bool)
        rows = torch.nonzero(hit).flatten()
        if op == "semi_join":
            return [_opaque(case["out"], rows), _opaque(case["out"], raw["p"][hit[raw["p"]]])]
        return [_opaque(case["out"], at[rows]), _opaque(case["out"], rows)]
    if op == "group":
        gr, ext = _groups(raw["k"])
        return [gr, ext, torch.zeros_like(ext).index_add_(0, gr, raw["m"])]
    if op == "star":
        in_dim = torch.zeros(case["keys"], dtype=torch.bool, device="cuda")
        in_dim[raw["l"]] = True
        rows = torch.nonzero((raw["filter"] < 400) & in_dim[raw["fk"]]).flatten()
        g = raw["gkey"][rows]
        gr, ext = _groups(g)
        sums = torch.zeros_like(ext).index_add_(0, gr, raw["measure"][rows])
        return [t.cpu().numpy().astype(np.uint64) for t in (g[ext], ext, sums)] + [rows.numel()]
    if op == "batch":
        consts = _batch_consts(case, raw)
        hit = [raw[i] < c for i, c in enumerate(consts)]
        return [np.array([int(h.sum().item()) for h in hit], np.uint64),
                np.array([int(raw[i][h].sum().item()) for i, h in enumerate(hit)], np.uint64)]
    v = raw["v"]
    hit = v < (1 << 20)
    return [_features(v), None, None, None, None, None, int(v[hit].sum().item()), int(hit.sum().item())]
