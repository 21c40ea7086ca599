"""COUNT(DISTINCT) beside DOUBLE aggregates: the distinct count lies in a
32-bit word of the shared state, next to the DOUBLE ops' 64-bit words, in
either order; shared tables, HBM tables, NULL keys and the INT64_MIN key
(shared states of their own at every estimate), on a handle, in a batch and in
a served query that runs alone.  Counts exact against the oracle, DOUBLE
within the oracle tests' relative tolerance."""
import numpy as np
import pytest

import oracle
from slothdb_gb300 import capi
from slothdb_gb300.capi import BIGINT, DOUBLE, INTEGER, SMALLINT, VARCHAR
from test_gpu_groupby import check
from util import compare, gpu_to_dict

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_lib", "gblib")]

# of (v, w, x): columns of distinct values, the DOUBLE column
AGGS = {
    "first": [("count_distinct", "v"), ("sum", "x"), ("avg", "x")],
    "between": [("sum", "x"), ("count_distinct", "v"), ("min", "x")],
    "last": [("max", "x"), ("avg", "x"), ("count_distinct", "v")],
    "two": [("count_distinct", "v"), ("max", "x"), ("count_distinct", "w"), ("count_star", None)],
    "two_first": [("count_distinct", "w"), ("count_distinct", "v"), ("sum", "x")],
}


def table(key, groups, n=60_007):
    """(types, group columns, columns, nulls without the DOUBLE's, column numbers)"""
    rng = np.random.default_rng(groups)
    k = rng.integers(0, groups, n)
    v = rng.integers(-40, 40, n).astype(np.int32)
    w = rng.integers(0, 10**9, n) // 10**7
    x = rng.normal(100, 25, n)
    at = lambda b: dict(v=b, w=b + 1, x=b + 2)  # noqa: E731
    rest = ([INTEGER, BIGINT, DOUBLE], [v, w, x])
    if key == "integer":
        return [INTEGER] + rest[0], [0], [k.astype(np.int32)] + rest[1], [None] * 4, at(1)
    if key == "bigint":  # NULL keys and the table's empty marker
        k = k * 10**12
        k[::97] = np.iinfo(np.int64).min
        return [BIGINT] + rest[0], [0], [k] + rest[1], [rng.random(n) < 0.1] + [None] * 3, at(1)
    if key == "pair":
        a, b = (k // 7).astype(np.int32), (k % 7).astype(np.int16)
        return [INTEGER, SMALLINT] + rest[0], [0, 1], [a, b] + rest[1], [None] * 5, at(2)
    text = [b"key-%d" % i for i in k]
    offs = np.zeros(n + 1, np.int64)
    np.cumsum([len(t) for t in text], out=offs[1:])
    return ([VARCHAR] + rest[0], [0], [(offs, np.frombuffer(b"".join(text), np.uint8).copy())] + rest[1], [None] * 4,
            at(1))


def named(aggs, at):
    return [(kind, at[c] if c else -1) for kind, c in aggs]


@pytest.mark.parametrize("est", [0, 900, 50_000])
@pytest.mark.parametrize("order", sorted(AGGS))
@pytest.mark.parametrize("key", ["integer", "bigint", "pair", "varchar"])
def test_handle(key, order, est):
    types, gcols, cols, nulls, at = table(key, 900)
    aggs = named(AGGS[order], at)
    has_nulls = any(m is not None for m in nulls)
    check(types, gcols, aggs, cols, nulls=nulls if has_nulls else None, est_groups=est, device=True)
    nulls = list(nulls)
    nulls[at["x"]] = np.random.default_rng(5).random(len(cols[at["x"]])) < 0.2
    check(types, gcols, aggs, cols, nulls=nulls, est_groups=est)
    if key != "varchar":  # more than one ingest into the same states, with a predicate
        check(types, gcols, aggs, cols, nulls=nulls, est_groups=est, chunks=19_968, filters=[(at["x"], "<", 110.0)])


def test_batch_and_lone_served_query():
    """The same queries in a batch (general tiles) and served with an estimate
    that makes them run alone."""
    import torch
    todo = []
    for key in ("integer", "bigint", "pair", "varchar"):
        types, gcols, cols, nulls, at = table(key, 300, n=20_011)
        for order in sorted(AGGS):
            todo.append((types, gcols, named(AGGS[order], at), cols, nulls))

    def dev(c):
        if isinstance(c, tuple):
            return tuple(torch.from_numpy(p).cuda() for p in c)
        return torch.from_numpy(np.ascontiguousarray(c)).cuda()

    def words(nulls):
        return [None if m is None else torch.from_numpy(capi.validity_words(~m).view(np.int64)).cuda() for m in nulls]

    b = capi.Batch()
    srv = capi.Server(budget_bytes=64 << 30)
    try:
        keep, tickets = [], []
        for types, gcols, aggs, cols, nulls in todo:
            d, vw, n = [dev(c) for c in cols], words(nulls), len(cols[-1])
            keep.append((d, vw))
            nullable = [i for i, m in enumerate(nulls) if m is not None]
            b.add(types, gcols, aggs, d, n, validity=vw, nullable=nullable, est_groups=300)
            tickets.append((srv.add_table(types, d, n, validity=vw), n, nullable))
        torch.cuda.synchronize()
        b.run()
        tickets = [srv.submit(t, 0, n, q[1], q[2], nullable=nullable, est_groups=1 << 20)
                   for (t, n, nullable), q in zip(tickets, todo)]
        for i, (types, gcols, aggs, cols, nulls) in enumerate(todo):
            want = oracle.run_query(types, gcols, aggs, cols, nulls=nulls)
            out = [types[c] for c in gcols] + [oracle.agg_out_type(oracle.AGG_NAMES[a], types[c] if c >= 0 else 0)
                                               for a, c in aggs]
            compare(gpu_to_dict(b.result(i), len(gcols), out), want)
            assert srv.wait(tickets[i])
            compare(gpu_to_dict(srv.result(tickets[i]), len(gcols), out), want)
    finally:
        srv.close()
        b.close()


def test_parquet_ingest():
    types, gcols, cols, _, at = table("integer", 900)
    aggs = named(AGGS["two_first"], at)
    from slothdb_gb300 import parquet as pq
    data = pq.write([pq.Column("k", pq.T_INT32, values=cols[0]), pq.Column("v", pq.T_INT32, values=cols[1]),
                     pq.Column("w", pq.T_INT64, values=cols[2]), pq.Column("x", pq.T_DOUBLE, values=cols[3])],
                    row_group_rows=20_000)
    want = oracle.run_query(types, gcols, aggs, cols)
    for est in (0, 50_000):
        pf = capi.ParquetFile(data)
        pf.upload()
        g = capi.GroupBy(types, gcols, aggs, est_groups=est)
        try:
            capi.ingest_parquet(g, pf, [0, 1, 2, 3], device=True)
            g.finalize()
            res = g.result()
        finally:
            g.close()
            pf.close()
        compare(gpu_to_dict(res, 1, [INTEGER, BIGINT, BIGINT, DOUBLE]), want)
