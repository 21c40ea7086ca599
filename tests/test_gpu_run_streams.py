"""Run tables of index streams of many lengths: around the windows of the short
walk (1,024 bytes) and the long one (8,192), around the line between them
(4,096 bytes), short and long ones in one file, beside level streams; and many
short streams in no more time than the same rows in long ones."""
import numpy as np
import pytest

import oracle
from slothdb_gb300 import capi
from slothdb_gb300 import parquet as pq
from slothdb_gb300.capi import BIGINT, INTEGER
from util import compare, gpu_to_dict

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_lib", "gblib")]

AGGS = [("count_star", -1), ("sum", 1), ("min", 1), ("max", 1)]


def run(data, device, profile=None):
    pf = capi.ParquetFile(data)
    if device:
        pf.upload()
    g = capi.GroupBy([INTEGER, BIGINT], [0], AGGS, est_groups=300)
    try:
        g.set_profiling(profile is not None)
        capi.ingest_parquet(g, pf, [0, 1], device=device)
        g.finalize()
        if profile is not None:
            profile.append(g.profile())
        return gpu_to_dict(g.result(), 1, [INTEGER, BIGINT, BIGINT, BIGINT, BIGINT])
    finally:
        g.close()
        pf.close()


def indices(kind, n, rng):
    pick = rng.integers(0, 256, n)
    if kind == "runs":  # a header every two bytes
        return np.repeat(pick, 9)[:n]
    if kind == "mixed":
        return np.repeat(pick, rng.integers(1, 30, n))[:n]
    return pick


@pytest.mark.parametrize("rows", [1, 7, 90, 500, 1000, 1010, 1030, 2040, 3200, 4060, 4075, 4090, 4110, 8170, 8200, 30_000])
@pytest.mark.parametrize("kind", ["packed", "runs", "mixed"])
def test_stream_lengths(kind, rows):
    n = min(60_007, 40 * rows + 13)
    rng = np.random.default_rng(rows)
    idx = indices(kind, n, rng).astype(np.uint32)
    d = rng.permutation(1 << 20)[:256].astype(np.int32)
    v = np.arange(n, dtype=np.int64)
    data = pq.write([pq.Column("k", pq.T_INT32, dictionary=d, indices=idx), pq.Column("v", pq.T_INT64, values=v)],
                    page_rows=rows, row_group_rows=25_000)
    orc = oracle.run_query([INTEGER, BIGINT], [0], AGGS, [d[idx], v])
    for device in (False, True):
        compare(run(data, device), orc)


@pytest.mark.parametrize("k_rows,v_rows", [(200, 20_000), (20_000, 200), (3000, 5000)])
def test_short_and_long_streams_in_one_file(k_rows, v_rows):
    n = 200_003
    rng = np.random.default_rng(k_rows)
    idx, vid = indices("mixed", n, rng).astype(np.uint32), rng.integers(0, 70_000, n).astype(np.uint32)
    d, dv = rng.permutation(1 << 20)[:256].astype(np.int32), rng.integers(0, 10**9, 70_000)
    data = pq.write([pq.Column("k", pq.T_INT32, dictionary=d, indices=idx, page_rows=k_rows),
                     pq.Column("v", pq.T_INT64, dictionary=dv, indices=vid, page_rows=v_rows)], row_group_rows=90_000)
    orc = oracle.run_query([INTEGER, BIGINT], [0], AGGS, [d[idx], dv[vid]])
    for device in (False, True):
        compare(run(data, device), orc)


def test_short_streams_cost_no_more_than_long_ones():
    """5,000 streams of 200 rows against 62 of 16,384 (the file in host memory:
    its run tables are made in each call): 1,024 threads for each of the short
    ones took 5 times as long."""
    n = 1_000_000
    rng = np.random.default_rng(1)
    idx = rng.integers(0, 256, n).astype(np.uint32)
    d, v = np.arange(256, dtype=np.int32), rng.integers(0, 10**6, n)
    best = []
    for rows in (200, 16_384):
        data = pq.write([pq.Column("k", pq.T_INT32, dictionary=d, indices=idx), pq.Column("v", pq.T_INT64, values=v)],
                        page_rows=rows)
        prof = []
        for _ in range(5):
            run(data, False, prof)
        best.append(min(p["k_pq_runs"][1] for p in prof))
    assert best[0] <= 2 * best[1], best
