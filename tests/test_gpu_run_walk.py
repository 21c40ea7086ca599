"""The run walk of dictionary-index streams around its 8 KB windows: streams
of short RLE runs (a header every 2 to 5 bytes), of RLE and bit-packed runs in
turn, of one packed run over many windows and of one RLE run, on pages of
several sizes; exact against the oracle."""
import numpy as np
import pytest

import oracle
from slothdb_gb300 import capi
from slothdb_gb300 import parquet as pq
from slothdb_gb300.capi import BIGINT, INTEGER
from util import compare, gpu_to_dict

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_lib", "gblib")]


def indices(kind, n, n_dict):
    rng = np.random.default_rng(n + n_dict)
    pick = rng.integers(0, n_dict, n).astype(np.uint32)
    if kind == "runs8":
        return np.repeat(pick, 8)[:n]
    if kind == "mixed":  # runs of 1 to 40
        return np.repeat(pick, rng.integers(1, 41, n))[:n]
    if kind == "packed":
        return pick
    return np.full(n, n_dict - 1, dtype=np.uint32)  # one run


@pytest.mark.parametrize("n_dict", [2, 200, 300, 70_000])
@pytest.mark.parametrize("kind", ["runs8", "mixed", "packed", "one"])
def test_run_walk(kind, n_dict):
    n = 140_001
    idx = indices(kind, n, n_dict)
    dictionary = np.random.default_rng(7).permutation(1 << 20)[:n_dict].astype(np.int32)
    v = np.arange(n, dtype=np.int64)
    aggs = [("count_star", -1), ("sum", 1), ("min", 1), ("max", 1)]
    orc = oracle.run_query([INTEGER, BIGINT], [0], aggs, [dictionary[idx], v])
    for page_rows in (n, 32_767, 4_099):
        data = pq.write([pq.Column("k", pq.T_INT32, dictionary=dictionary, indices=idx),
                         pq.Column("v", pq.T_INT64, values=v)], row_group_rows=n, page_rows=page_rows)
        pf = capi.ParquetFile(data)
        pf.upload()
        g = capi.GroupBy([INTEGER, BIGINT], [0], aggs, est_groups=n_dict)
        try:
            capi.ingest_parquet(g, pf, [0, 1], device=True)
            g.finalize()
            res = g.result()
        finally:
            g.close()
            pf.close()
        compare(gpu_to_dict(res, 1, [INTEGER, BIGINT, BIGINT, BIGINT, BIGINT]), orc)
