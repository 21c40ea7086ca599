"""The work that users of the GROUP BY path have it do, as measurable cases.

Every case goes through the public binding (``slothdb_gb300.capi``): one
GROUP BY handle over device or host columns (``hash`` and ``radix``), one
over a Parquet file resident in HBM or held in host memory (``parquet``), many
queries run together (``batch``) and a burst of queries to the server
(``serve``).  A handle, a batch and a server are what a program keeps between
calls, so ``prepare`` makes them; ``run`` rewinds, feeds, finishes and takes
the result.  A GROUP BY returns its groups in no order, so ``run`` puts them
the way a program does that joins them to its own table: each group's row goes
to the place its key stands for there (groups without rows keep zeros), small
results on the host, large ones on the GPU.  A string key begins with four
characters that number it, as codes and names with a number do.
"""
import ctypes

import numpy as np
import torch

from slothdb_gb300 import capi, datagen, parquet

M31 = (1 << 31) - 1
SPREAD = 0x5DEECE6D  # odd: key -> key * SPREAD mod 2^31 is one to one
SPREAD_BACK = pow(SPREAD, -1, 1 << 31)
HOST_GROUPS = 8192  # results up to this many groups are taken and placed on the host


# ------------------------------------------------------------------- cases
def listed():
    return [
        # one chunk of the engine's vectors (DataChunk of 2,048 rows) from host memory: the smallest call
        dict(name="chunk_2k", kind="hash", key="int32", rows=2048, groups=64, aggs="int4", spread=False, est=64,
             nulls=False, select=1.0, mem="host"),
        # the plain GROUP BY of the benchmark: 1M rows, 1,024 keys, COUNT/SUM/MIN/MAX
        dict(name="plain_1m", kind="hash", key="int32", rows=1_000_000, groups=1024, aggs="int4", spread=False,
             est=1024, nulls=False, select=1.0, mem="device"),
        # a measure column of DOUBLEs with NULLs, a BIGINT key with NULLs, a WHERE that keeps half; odd row count
        dict(name="nulls_3m", kind="hash", key="int64", rows=3_000_017, groups=5000, aggs="avg", spread=True,
             est=5000, nulls=True, select=0.5, mem="device"),
        # composite (INTEGER, SMALLINT) key with more groups than a block's shared memory holds
        dict(name="pair_10m", kind="hash", key="pair", rows=10_000_000, groups=300_000, aggs="sum_max", spread=False,
             est=300_000, nulls=False, select=1.0, mem="device"),
        # names or codes as keys: strings of 8 to 32 characters
        dict(name="varchar_4m", kind="hash", key="varchar", rows=4_000_000, groups=30_000, aggs="sum_max",
             spread=False, est=30_000, nulls=False, select=1.0, mem="device"),
        # COUNT(DISTINCT visitor) per item
        dict(name="distinct_20m", kind="hash", key="int32", rows=20_000_000, groups=100_000, aggs="distinct",
             spread=True, est=100_000, nulls=False, select=1.0, mem="device"),
        # the headline: 100M rows, Zipf(1.1) over 20M BIGINT keys, COUNT/SUM/AVG, the ten most frequent
        dict(name="zipf_100m", kind="radix", rows=100_000_000, values=20_000_000, aggs="avg", limit=10, select=1.0),
        # fused decode + filter + aggregate of a resident file, as the 200M-row benchmark's but smaller
        dict(name="parquet_32m", kind="parquet", rows=32_000_000, dict=65_536, codec="none", select=0.1,
             group_rows=1_000_000, mem="device"),
        # the same file compressed, with the two codecs in use
        dict(name="parquet_snappy_8m", kind="parquet", rows=8_000_000, dict=65_536, codec="snappy", select=0.1,
             group_rows=1_000_000, mem="device"),
        dict(name="parquet_zstd_8m", kind="parquet", rows=8_000_000, dict=65_536, codec="zstd", select=0.1,
             group_rows=1_000_000, mem="device"),
        # independent queries over uneven tables in one submission (a dashboard)
        dict(name="batch_16", kind="batch", tables=16, shapes=3, rows_lo=5.0, rows_hi=7.0, groups_hi=5.0, varchar=0.25),
        # a burst of queries of different sizes over resident tables
        dict(name="serve_32", kind="serve", queries=32, shapes=4, rows_hi=7.5),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["hash"] * 5 + ["radix"] + ["parquet"] * 3 + ["batch", "serve"])
    if kind == "hash":
        key = rng.choice(["int32", "int64", "pair", "varchar"])
        rows = _log(rng, 500, 4_000_000 if key == "varchar" else 20_000_000)
        groups = max(1, min(_log(rng, 2, 500_000), rows // 2))
        aggs = rng.choice(["int4", "sum_max", "avg", "distinct"])
        return dict(kind=kind, key=key, rows=rows, groups=groups, aggs=aggs, spread=rng.random() < 0.5,
                    est=groups if rng.random() < 0.8 else 0, nulls=rng.random() < 0.3,
                    select=1.0 if rng.random() < 0.6 else round(rng.uniform(0.01, 0.99), 3),
                    mem="host" if rng.random() < 0.2 else "device")
    if kind == "radix":
        rows = _log(rng, 4_000_000, 90_000_000)
        return dict(kind=kind, rows=rows, values=_log(rng, 300_000, max(300_000, rows // 5)),
                    aggs=rng.choice(["avg", "sum_max"]), limit=rng.choice([10, 100, 1000]),
                    select=1.0 if rng.random() < 0.6 else round(rng.uniform(0.05, 0.99), 3))
    if kind == "parquet":
        codec = rng.choice(["none", "snappy", "zstd"])
        return dict(kind=kind, rows=_log(rng, 20_000, 24_000_000 if codec == "none" else 6_000_000),
                    dict=_log(rng, 100, 65_536), codec=codec, select=round(rng.uniform(0.01, 1.0), 3),
                    group_rows=rng.choice([122_880, 500_000, 1_000_000]),
                    mem="host" if rng.random() < 0.2 else "device")
    if kind == "batch":
        return dict(kind=kind, tables=rng.randint(4, 16), shapes=rng.randint(5, 10_000),
                    rows_lo=round(rng.uniform(4.0, 5.0), 2),
                    rows_hi=round(rng.uniform(5.0, 6.9), 2), groups_hi=round(rng.uniform(3.0, 5.0), 2),
                    varchar=rng.choice([0.0, 0.25, 0.5]))
    return dict(kind=kind, queries=rng.randint(4, 32), shapes=rng.randint(5, 10_000),
                rows_hi=round(rng.uniform(5.0, 7.4), 2))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ints(g, lo, hi, n, dtype=torch.int64):
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=torch.int64).to(dtype)


def _words(valid):
    """Validity words of a device bool column."""
    n = valid.numel()
    v = torch.zeros((n + 63) // 64 * 64, dtype=torch.int64, device="cuda")
    v[:n] = valid
    return (v.view(-1, 64) << torch.arange(64, device="cuda")).sum(1)


def _pool(groups, seed):
    """Distinct strings of 8 to 32 characters (offsets, bytes), on the host; the first four characters number them."""
    rng = np.random.default_rng(seed)
    offs, data = datagen.varchar_pool(groups, rng)
    data = data.copy()
    num = np.arange(groups)
    for j in range(4):
        data[offs[:-1] + j] = datagen.ALNUM[num % 36]
        num //= 36
    return offs, data


def _pick_strings(offs, data, pick):
    offs, data = torch.from_numpy(offs).cuda(), torch.from_numpy(data).cuda()
    lens = (offs[1:] - offs[:-1])[pick]
    out = torch.zeros(pick.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=out[1:])
    total = int(out[-1])
    at = torch.repeat_interleave(offs[pick] - out[:-1], lens, output_size=total)
    return out, data[at + torch.arange(total, device="cuda")]


AGGS = {  # (aggregates over the column numbers from `first` on, types of those columns)
    "int4": lambda c: ([("count_star", -1), ("sum", c), ("min", c), ("max", c)], [capi.BIGINT]),
    "sum_max": lambda c: ([("count_star", -1), ("sum", c), ("max", c + 1)], [capi.BIGINT, capi.INTEGER]),
    "avg": lambda c: ([("count_star", -1), ("count", c), ("sum", c), ("avg", c)], [capi.DOUBLE]),
    "distinct": lambda c: ([("count_distinct", c), ("count_star", -1)], [capi.INTEGER]),
}


def _hash_data(case, seed):
    """Columns of a hash case on the GPU: group number of each row, key columns, value columns, filter column, NULLs."""
    g, n, groups = _gen(seed), case["rows"], case["groups"]
    gid = _ints(g, 0, groups, n)
    pool = None
    if case["key"] == "varchar":
        pool = _pool(groups, seed)
        keys, ktypes = [_pick_strings(*pool, gid)], [capi.VARCHAR]
    elif case["key"] == "pair":
        keys, ktypes = [(gid >> 6).to(torch.int32), (gid & 63).to(torch.int16)], [capi.INTEGER, capi.SMALLINT]
    else:
        k = (gid * SPREAD) & M31 if case["spread"] else gid
        wide = case["key"] == "int64"
        keys, ktypes = [k if wide else k.to(torch.int32)], [capi.BIGINT if wide else capi.INTEGER]
    aggs, vtypes = AGGS[case["aggs"]](len(keys))
    vals = []
    for t in vtypes:
        if t == capi.DOUBLE:
            vals.append(torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * 25 + 100)
        elif t == capi.BIGINT:
            vals.append(_ints(g, 0, 10**6, n))
        else:
            vals.append(_ints(g, 0, 2000, n, torch.int32) if case["aggs"] == "distinct" else
                        _ints(g, -(2**31), M31, n, torch.int32))
    types = ktypes + vtypes
    cols = keys + vals
    filters = []
    if case["select"] < 1.0:
        filters = [(len(cols), "<", int(case["select"] * 1000))]
        cols.append(_ints(g, 0, 1000, n, torch.int16))
        types.append(capi.SMALLINT)
    valid = [None] * len(cols)
    if case["nulls"]:
        where = [len(keys)] if case["key"] != "int64" else [0, len(keys)]
        for c in where:
            valid[c] = torch.rand(n, generator=g, device="cuda") >= 0.05
    return dict(gid=gid, pool=pool, cols=cols, types=types, group_cols=list(range(len(keys))), aggs=aggs,
                filters=filters, valid=valid)


def _host(t):
    return (t[0].cpu().numpy(), t[1].cpu().numpy()) if isinstance(t, tuple) else t.cpu().numpy()


def _prepare_hash(case, seed):
    d = _hash_data(case, seed)
    words = [None if v is None else _words(v) for v in d["valid"]]
    cols = d["cols"]
    if case["mem"] == "host":
        cols = [_host(c) for c in cols]
        words = [None if w is None else w.cpu().numpy().view(np.uint64) for w in words]
    h = capi.GroupBy(d["types"], d["group_cols"], d["aggs"], filters=d["filters"], est_groups=case["est"],
                     nullable=[c for c, w in enumerate(words) if w is not None])
    return dict(case=case, h=h, cols=cols, words=words if any(w is not None for w in words) else None,
                tables=_tables())


def _zipf_cdf(n):
    c = torch.cumsum(torch.arange(1, n + 1, device="cuda", dtype=torch.float64) ** -1.1, 0)
    return c / c[-1]


def _radix_data(case, seed):
    g, n = _gen(seed), case["rows"]
    cdf = _zipf_cdf(case["values"])
    k = torch.empty(n, dtype=torch.int64, device="cuda")
    for lo in range(0, n, 1 << 25):
        hi = min(n, lo + (1 << 25))
        r = torch.searchsorted(cdf, torch.rand(hi - lo, generator=g, device="cuda", dtype=torch.float64), right=True)
        # ranks spread over [0, 2^40) by an odd multiplier
        k[lo:hi] = (r.clamp_(max=case["values"] - 1) * 0x9E3779B97F4A7C15) & ((1 << 40) - 1)
    if case["aggs"] == "avg":
        vals = [torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * 25 + 100]
        below = torch.special.ndtri(torch.tensor(case["select"], dtype=torch.float64))
        filters = [(1, "<", 100.0 + 25.0 * float(below))]
        types, aggs = [capi.BIGINT, capi.DOUBLE], [("count_star", -1), ("sum", 1), ("avg", 1)]
    else:
        vals = [_ints(g, 0, 10**6, n), _ints(g, -(2**31), M31, n, torch.int32)]
        filters = [(1, "<", int(case["select"] * 10**6))]
        types, aggs = [capi.BIGINT, capi.BIGINT, capi.INTEGER], [("count_star", -1), ("sum", 1), ("max", 2)]
    return k, vals, types, aggs, filters if case["select"] < 1.0 else []


def _prepare_radix(case, seed):
    k, vals, types, aggs, filters = _radix_data(case, seed)
    h = capi.GroupBy(types, [0], aggs, filters=filters, est_groups=case["rows"] // 12)
    h.set_topn(1, False, case["limit"])
    return dict(case=case, h=h, cols=[k] + vals, words=None)


def _prepare_parquet(case, seed):
    data = _parquet_data(case, seed)[0]
    data = np.frombuffer(data, dtype=np.uint8)
    pin = capi.PinnedBuffer(len(data))  # a program reads the file into page-locked memory
    pin.view(np.uint8)[:] = data
    pf = capi.ParquetFile(pin.view(np.uint8))
    if case["mem"] == "device":
        pf.upload()
    h = capi.GroupBy([capi.INTEGER, capi.SMALLINT, capi.BIGINT], [0], [("sum", 2), ("count_star", -1)],
                     filters=[(1, "<", int(case["select"] * 1000))], est_groups=case["dict"])
    # the program's own table of the keys (the file's dictionary, drawn first)
    names = np.unique(np.random.default_rng(seed).integers(0, 2**31, case["dict"], dtype=np.int64).astype(np.int32))
    return dict(case=case, h=h, pf=pf, pin=pin, names=torch.from_numpy(names).cuda())


def _parquet_data(case, seed):
    return parquet.filter_groupby_file(n_rows=case["rows"], seed=seed, n_dict=case["dict"],
                                       row_group_rows=case["group_rows"],
                                       codec=None if case["codec"] == "none" else case["codec"])


def _batch_shapes(case, seed):
    s = datagen.batch_shapes(case["tables"], seed=case["shapes"], rows_exp=(case["rows_lo"], case["rows_hi"]),
                             groups_exp=(2.0, case["groups_hi"]), varchar_frac=case["varchar"])
    return [dict(x, seed=seed * 100_003 + i) for i, x in enumerate(s)]


def _string_table(n, groups, seed):
    g = _gen(seed)
    return [_pick_strings(*_pool(groups, seed), _ints(g, 0, groups, n)), _ints(g, 0, 10**6, n),
            _ints(g, -(2**31), M31, n, torch.int32)]


def _prepare_batch(case, seed):
    shapes, b, n, names = _batch_shapes(case, seed), capi.Batch(), 0, 0
    sizes = {"composite": [], "varchar": []}
    for i, s in enumerate(shapes):
        pair = s["kind"] == "composite"
        q = datagen.BATCH_COMPOSITE if pair else datagen.BATCH_VARCHAR
        cols = datagen.batch_table_device(s) if pair else _string_table(s["rows"], s["groups"], s["seed"])
        b.add(q["col_types"], q["group_cols"], q["aggs"], cols, s["rows"], est_groups=s["groups"])
        sizes[s["kind"]].append((i, n if pair else names))
        if pair:
            n += (max(1, s["groups"] // 64)) * 64
        else:
            names += s["groups"]
    first = torch.tensor([p for _, p in sizes["varchar"]]).cuda()
    return dict(case=case, b=b, places=n, names=names, first=first, sizes=sizes, tables=_tables())


SERVED = [("plain", 50_000_000, 1024), ("filter", 50_000_000, 4096), ("composite", 40_000_000, 10_000),
          ("varchar", 10_000_000, 1000)]


def _served_table(i, seed):
    kind, n, groups = SERVED[i]
    g = _gen(seed * 10 + i)
    if kind == "plain":
        return [_ints(g, 0, groups, n, torch.int32), _ints(g, 0, 10**6, n)]
    if kind == "filter":
        runs = _ints(g, 0, groups, n // 4 + 1)
        return [((torch.repeat_interleave(runs, 4)[:n] * SPREAD) & M31).to(torch.int32),
                _ints(g, 0, 1000, n, torch.int16), _ints(g, -10**9, 10**9, n)]
    if kind == "composite":
        gid = _ints(g, 0, groups, n)
        return [(gid >> 6).to(torch.int32), (gid & 63).to(torch.int16), _ints(g, 0, 10**6, n),
                _ints(g, -(2**31), M31, n, torch.int32)]
    return _string_table(n, groups, seed * 10 + i)


def _served_queries(case):
    rng, out = np.random.default_rng(case["shapes"]), []
    for _ in range(case["queries"]):
        t = int(rng.integers(0, 4))
        kind, n, groups = SERVED[t]
        rows = min(n, int(10 ** rng.uniform(4, case["rows_hi"])))
        r0 = int(rng.integers(0, n - rows + 1)) // 64 * 64
        sel = float(rng.uniform(0.01, 1.0))
        q = {"plain": dict(group_cols=[0], aggs=[("count_star", -1), ("sum", 1), ("min", 1), ("max", 1)],
                           filters=[(1, "<", int(sel * 10**6))]),
             "filter": dict(group_cols=[0], aggs=[("sum", 2), ("count_star", -1)], filters=[(1, "<", int(sel * 1000))]),
             "composite": dict(group_cols=[0, 1], aggs=datagen.BATCH_COMPOSITE["aggs"],
                               filters=[(2, "<", int(sel * 10**6))]),
             "varchar": dict(group_cols=[0], aggs=datagen.BATCH_VARCHAR["aggs"], filters=[(1, "<", int(sel * 10**6))])}
        out.append(dict(q[kind], table=t, row_begin=r0, row_end=r0 + rows, est_groups=groups))
    return out


def _prepare_serve(case, seed):
    s = capi.Server(40 << 30)
    for i, (kind, n, _) in enumerate(SERVED):
        s.add_table(datagen.SERVE_TYPES[kind], _served_table(i, seed), n)
    torch.cuda.synchronize()  # the server's own threads read the tables
    return dict(case=case, server=s, queries=_served_queries(case))


def prepare(case, seed):
    capi.load(build_if_missing=True)
    return {"hash": _prepare_hash, "radix": _prepare_radix, "parquet": _prepare_parquet, "batch": _prepare_batch,
            "serve": _prepare_serve}[case["kind"]](case, seed)


# ----------------------------------------------------------------- results
class _Pointer:
    def __init__(self, ptr, n, kind):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=(n,), typestr=kind, version=3)


KINDS = {capi.SMALLINT: "<i2", capi.INTEGER: "<i4", capi.BIGINT: "<i8", capi.DOUBLE: "<f8"}


def _view(ptr, n, kind):
    return torch.as_tensor(_Pointer(ptr, n, kind), device="cuda")


def _valid_bits(r, c, n):
    w = _view(r.validity[c], (n + 63) // 64, "<i8")
    return ((w[:, None] >> torch.arange(64, device="cuda")) & 1).view(-1)[:n]


def _device_columns(r):
    n = int(r.n_rows)
    return n, [None if r.types[c] == capi.VARCHAR else _view(r.data[c], n, KINDS[r.types[c]]) for c in range(r.n_cols)]


def _place(idx, col, places):
    return torch.zeros(places, dtype=col.dtype, device="cuda").scatter_(0, idx, col)


def _place_host(idx, col, places):
    out = np.zeros(places, dtype=col.dtype)
    out[idx] = col
    return out


DIGIT = np.zeros(256, dtype=np.int64)
DIGIT[datagen.ALNUM] = np.arange(36)
PLACE = 36 ** np.arange(4)


def _tables():
    return torch.from_numpy(DIGIT).cuda(), torch.from_numpy(PLACE).cuda()


def _by_string(text, first, places, tables):
    """Device results of a VARCHAR key, each (offsets, bytes, other columns), by the strings' numbers: result i's from
    place first[i] on."""
    at = torch.arange(32, device="cuda")
    data, offs, ends = text[0][1], text[0][0][:-1], text[0][0][1:]
    cols = text[0][2]
    if len(text) > 1:
        n = torch.tensor([[t[0].numel() - 1, t[1].numel()] for t in text]).cuda()
        base = (torch.cumsum(n[:, 1], 0) - n[:, 1]).repeat_interleave(n[:, 0])
        first = first.repeat_interleave(n[:, 0])
        data = torch.cat([t[1] for t in text])
        offs, ends = torch.cat([t[0][:-1] for t in text]) + base, torch.cat([t[0][1:] for t in text]) + base
        cols = [torch.cat([t[2][c] for t in text]) for c in range(len(cols))]
    spots = offs[:, None] + at
    chars = data[torch.where(spots < ends[:, None], spots, offs[:, None])]
    idx = tables[0][chars[:, :4].long()].mul_(tables[1]).sum(1) + first
    out = torch.zeros((places, 32), dtype=torch.uint8, device="cuda")
    out[idx] = chars  # beyond a string's end: its first character
    return [out] + [_place(idx, c, places) for c in [ends - offs] + cols]


def _text(r, cols):
    offs = _view(r.offsets[0], int(r.n_rows) + 1, "<i8")
    return offs, _view(r.data[0], int(offs[-1]), "|u1"), cols


def _host_strings(names, places):
    """Places of the strings by their numbers, and their characters there."""
    k = names.astype("S32")
    text = k.view(np.uint8).reshape(-1, 32)
    idx = DIGIT[text[:, :4]] @ PLACE
    return idx, _place_host(idx, k, places).view(np.uint8)


def _hash_result(case, h, tables):
    nk, nulls, groups = 2 if case["key"] == "pair" else 1, case["nulls"], case["groups"]
    if groups <= HOST_GROUPS:
        res = h.result()
        cols = [v for v, _ in res[nk:]] + ([ok for _, ok in res[nk:]] if nulls else [])
        if case["key"] == "varchar":
            idx, text = _host_strings(res[0][0], groups)
            return [_place_host(idx, c, groups) for c in cols] + [text]
        k = res[0][0].astype(np.int64)
        idx = k * 64 + res[1][0] if nk == 2 else (k * SPREAD_BACK) & M31 if case["spread"] else k
        if nulls:
            idx = np.where(res[0][1], idx, groups)
        return [_place_host(idx, c, groups + 1) for c in cols]
    r = capi.Result()
    capi.check(h.lib.gb_agg_result_device(h.h, ctypes.byref(r)))
    n, cols = _device_columns(r)
    valid = [_valid_bits(r, c, n) for c in range(nk, r.n_cols)] if nulls else []
    if case["key"] == "varchar":
        return _by_string([_text(r, cols[1:] + valid)], 0, groups, tables)
    k = cols[0].long()
    idx = k * 64 + cols[1] if nk == 2 else (k * SPREAD_BACK) & M31 if case["spread"] else k
    if nulls:
        idx = torch.where(_valid_bits(r, 0, n) == 1, idx, groups)
    return [_place(idx, c, groups + 1) for c in cols[nk:] + valid]


def _run_hash(s):
    h = s["h"]
    h.reset()
    h.ingest(s["cols"], nrows=s["case"]["rows"], validity=s["words"], device=s["case"]["mem"] == "device")
    h.finalize()
    return _hash_result(s["case"], h, s["tables"])


def _run_radix(s):
    h = s["h"]
    h.reset()
    h.ingest(s["cols"], nrows=s["case"]["rows"], device=True)
    h.finalize()
    return [v for v, _ in h.result()]  # LIMIT rows, best first


def _run_parquet(s):
    h = s["h"]
    h.reset()
    capi.ingest_parquet(h, s["pf"], [0, 1, 2], device=s["case"]["mem"] == "device")
    h.finalize()
    r = capi.Result()
    capi.check(h.lib.gb_agg_result_device(h.h, ctypes.byref(r)))
    _, cols = _device_columns(r)
    idx = torch.searchsorted(s["names"], cols[0])
    return [_place(idx, c, s["case"]["dict"]) for c in cols]


def _run_batch(s):
    b = s["b"]
    b.run()
    results = {}
    for kind, where in s["sizes"].items():
        for i, _ in where:
            r = capi.Result()
            capi.check(b.lib.gb_batch_result_device(b.h, i, ctypes.byref(r)))
            results[i] = (r,) + _device_columns(r)
    out = {}
    if s["sizes"]["composite"]:
        got = [(results[i], base) for i, base in s["sizes"]["composite"]]
        cols = [torch.cat([x[2][c] for x, _ in got]) for c in range(5)]
        base = torch.tensor([p for _, p in got]).cuda().repeat_interleave(
            torch.tensor([x[1] for x, _ in got]).cuda(), output_size=cols[0].numel())
        idx = cols[0].long() * 64 + cols[1] + base
        out["pairs"] = [_place(idx, c, s["places"]) for c in cols[2:]]
    if s["sizes"]["varchar"]:
        where = s["sizes"]["varchar"]
        out["strings"] = _by_string([_text(results[i][0], results[i][2][1:]) for i, _ in where], s["first"], s["names"],
                                    s["tables"])
    return out


def _run_serve(s):
    srv = s["server"]
    tickets = [srv.submit(**q) for q in s["queries"]]
    text, vals = [], []
    for q, t in zip(s["queries"], tickets):
        srv.wait(t)
        res = srv.result(t)
        srv.release(t)
        nk, (kind, _, groups) = len(q["group_cols"]), SERVED[q["table"]]
        cols = [v.astype(np.int64) for v, _ in res[nk:]]
        if kind == "varchar":
            idx, names = _host_strings(res[0][0], groups)
            text.append(names)
        else:
            k = res[0][0].astype(np.int64)
            idx = k * 64 + res[1][0] if nk == 2 else (k * SPREAD_BACK) & M31 if kind == "filter" else k
        vals += [_place_host(idx, c, groups) for c in cols]
    return [np.concatenate(x) for x in (text, vals) if x]


def run(state):
    return {"hash": _run_hash, "radix": _run_radix, "parquet": _run_parquet, "batch": _run_batch,
            "serve": _run_serve}[state["case"]["kind"]](state)


# -------------------------------------------------------------------- work
WIDTH = {capi.SMALLINT: 2, capi.INTEGER: 4, capi.BIGINT: 8, capi.DOUBLE: 8}
STRING = 8 + 20  # an offset and the mean string


def work(case):
    n = case.get("rows", 0)
    if case["kind"] == "hash":
        keys = {"int32": [4], "int64": [8], "pair": [4, 2], "varchar": [STRING]}[case["key"]]
        aggs, vtypes = AGGS[case["aggs"]](len(keys))
        row = sum(keys) + sum(WIDTH[t] for t in vtypes) + (2 if case["select"] < 1.0 else 0)
        row += 0.125 * (1 + (case["key"] == "int64")) if case["nulls"] else 0
        return dict(bytes=n * row + case["groups"] * (sum(keys) + 8 * len(aggs)), flops=n * len(aggs))
    if case["kind"] == "radix":
        return dict(bytes=n * (16 if case["aggs"] == "avg" else 20) + case["limit"] * 32, flops=2 * n)
    if case["kind"] == "parquet":
        # the pages: indices of 16 bits in runs of four or so, 4-byte and 8-byte PLAIN values
        return dict(bytes=n * 14.0 + case["dict"] * 20, flops=2 * n)
    if case["kind"] == "batch":
        shapes = _batch_shapes(case, 0)
        return dict(bytes=sum(s["rows"] * (18 if s["kind"] == "composite" else STRING + 12) + s["groups"] * 28
                              for s in shapes), flops=sum(2 * s["rows"] for s in shapes))
    row = {"plain": 12, "filter": 14, "composite": 18, "varchar": STRING + 12}
    b = sum((q["row_end"] - q["row_begin"]) * row[SERVED[q["table"]][0]] + SERVED[q["table"]][2] * 32
            for q in _served_queries(case))
    return dict(bytes=b, flops=b / 8)


# ------------------------------------------------------------ exact results
def _sums(idx, x, places):
    return torch.zeros(places, dtype=x.dtype, device="cuda").index_add_(0, idx, x)


def exact(case, seed):
    """The DOUBLE aggregates in 64 bits from plain torch; everything else here is whole numbers."""
    if case["kind"] == "radix" and case["aggs"] == "avg":
        k, (x,), _, _, filters = _radix_data(case, seed)
        if filters:
            keep = x < filters[0][2]
            k, x = k[keep], x[keep]
        keys, inv, count = torch.unique(k, return_inverse=True, return_counts=True)
        best = torch.sort(count, descending=True, stable=True)[1][:case["limit"]]  # ties: smaller key first
        total = _sums(inv, x, keys.numel())[best]
        return [keys[best].cpu(), count[best].cpu(), total.cpu(), (total / count[best]).cpu()]
    if case["kind"] == "hash" and case["aggs"] == "avg" and case["key"] != "varchar":
        d, groups = _hash_data(case, seed), case["groups"]
        nk = len(d["group_cols"])
        idx, x = d["gid"], d["cols"][nk]
        if d["valid"][0] is not None:
            idx = torch.where(d["valid"][0], idx, groups)
        ok = d["valid"][nk] if d["valid"][nk] is not None else torch.ones_like(idx, dtype=torch.bool)
        if d["filters"]:
            keep = d["cols"][d["filters"][0][0]] < d["filters"][0][2]
            idx, x, ok = idx[keep], x[keep], ok[keep]
        total = _sums(idx, torch.where(ok, x, 0.0), groups + 1)
        count = _sums(idx, ok.long(), groups + 1)
        mean = torch.where(count > 0, total / count.clamp(min=1), 0.0)
        return [None, None, total, mean]
    return None
