"""Page decompression on the GPU (a block of threads per page): every byte
of a page reaches a group of its own row number modulo 1009, so a wrong or
misplaced byte changes a SUM, MIN or MAX; exact against the oracle."""
import os
import sys

import numpy as np
import pytest

import oracle
from slothdb_gb300 import capi
from slothdb_gb300 import parquet as pq
from slothdb_gb300.capi import BIGINT, INTEGER
from util import compare, gpu_to_dict

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import make_page_files as pages  # noqa: E402
from make_pyarrow_files import load  # noqa: E402

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_lib", "gblib")]

TYPES = [INTEGER, BIGINT]
AGGS = [("sum", 1), ("min", 1), ("max", 1), ("count_star", -1)]


def check(data, k, v):
    orc = oracle.run_query(TYPES, [0], AGGS, [k, v])
    for device in (False, True):
        pf = capi.ParquetFile(data)
        if device:
            pf.upload()
        g = capi.GroupBy(TYPES, [0], AGGS, est_groups=1009)
        try:
            capi.ingest_parquet(g, pf, [0, 1], device=device)
            g.finalize()
            res = g.result()
        finally:
            g.close()
            pf.close()
        compare(gpu_to_dict(res, 1, [INTEGER, BIGINT, BIGINT, BIGINT, BIGINT]), orc)


def values(kind, n):
    rng = np.random.default_rng(n)
    return {
        "random": lambda: rng.integers(-2**42, 2**42, n),            # literals longer than a window
        "zeros": lambda: np.zeros(n),                                 # one run: copies that overlap themselves
        "period": lambda: np.resize(np.array([5, -9, 2**41]), n),
        "small": lambda: rng.integers(0, 300, n),                     # short elements, long chains in a window
        "steps": lambda: np.repeat(rng.integers(0, 2**40, n // 50 + 1), 50)[:n],
        "far": lambda: np.resize(rng.integers(0, 2**42, 7001), n),    # copies from 56,008 bytes back
    }[kind]().astype(np.int64)


# v pages of 8n bytes around the window (8,192 bytes), the parsed piece (4,096
# compressed bytes), a block of a frame (131,072 bytes) and several of them
@pytest.mark.parametrize("n", [1, 3, 511, 512, 513, 1023, 1024, 1025, 16_383, 16_384, 16_385, 40_000])
@pytest.mark.parametrize("codec", ["snappy", "zstd"])
def test_page_sizes_and_patterns(codec, n):
    for kind in ("random", "zeros", "period", "small", "steps", "far"):
        v = values(kind, n)
        k = (np.arange(n) % 1009).astype(np.int32)
        check(pq.write([pq.Column("k", pq.T_INT32, values=k), pq.Column("v", pq.T_INT64, values=v)], page_rows=n,
                       codec=codec), k, v)


@pytest.mark.parametrize("name", sorted(pages.FILES))
def test_large_pages_of_pyarrow(name):
    k, v = pages.columns()
    check(load(name), k, v)
