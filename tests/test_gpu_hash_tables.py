"""The hash pipeline's tables around the sizes where its rules change: shared
tables of a few slots to none, HBM tables of an estimate at and past the
sparse sizes, estimates far off both ways; integers exact against the oracle,
DOUBLE within the oracle tests' relative tolerance."""
import numpy as np
import pytest

import oracle
from slothdb_gb300 import capi
from slothdb_gb300.capi import BIGINT, INTEGER, SMALLINT
from util import compare, gpu_to_dict

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_lib", "gblib")]

AGGS = [("count_star", -1), ("sum", 1), ("min", 1), ("max", 2)]


def run(types, keys, aggs, cols, est, filters=(), device=True, nulls=None, options=None):
    import torch
    nulls = nulls or [None] * len(cols)
    words = [None if m is None else capi.validity_words(~m) for m in nulls]
    nullable = [i for i, m in enumerate(nulls) if m is not None]
    g = capi.GroupBy(types, keys, aggs, filters=filters, nullable=nullable, est_groups=est, options=options)
    try:
        if device:
            cols = [torch.from_numpy(c).cuda() for c in cols]
            words = [None if w is None else torch.from_numpy(w.view(np.int64)).cuda() for w in words]
            torch.cuda.synchronize()
        for _ in range(2):  # a handle is run again after its reset
            g.reset()
            g.ingest(cols, nrows=len(cols[0]), validity=words if nullable else None, device=device)
            g.finalize()
        res = g.result()
    finally:
        g.close()
    out = [types[k] for k in keys] + [oracle.agg_out_type(oracle.AGG_NAMES[k], types[c] if c >= 0 else 0)
                                      for k, c in aggs]
    return gpu_to_dict(res, len(keys), out)


@pytest.mark.parametrize("groups", [1, 2, 127, 129, 2047, 2049, 4097, 8191, 8193, 65_537])
@pytest.mark.parametrize("est", ["right", "none", "low"])
def test_table_sizes(groups, est):
    n = 3 * groups + 70_001
    rng = np.random.default_rng(groups)
    k = (rng.integers(0, groups, n) * 2654435761 % (1 << 31)).astype(np.int32)
    v = rng.integers(-10**9, 10**9, n)
    m = rng.integers(-2**31, 2**31 - 1, n).astype(np.int32)
    types = [INTEGER, BIGINT, INTEGER]
    e = {"right": groups, "none": 0, "low": max(1, groups // 50)}[est]
    compare(run(types, [0], AGGS, [k, v, m], e), oracle.run_query(types, [0], AGGS, [k, v, m]))


@pytest.mark.parametrize("spread", ["stride", "high", "negative"])
def test_keys_of_one_residue(spread):
    """Keys that agree in their low or high bits, for the shared table's hash."""
    base = np.arange(1500, dtype=np.int64)
    k = {"stride": base << 20, "high": (base << 44) | 5, "negative": -(base << 32) - 1}[spread]
    rng = np.random.default_rng(3)
    k = k[rng.integers(0, 1500, 50_003)]
    v = rng.integers(0, 10**6, len(k))
    s = rng.integers(-100, 100, len(k)).astype(np.int16)
    types = [BIGINT, BIGINT, SMALLINT]
    compare(run(types, [0], AGGS, [k, v, s], 1500), oracle.run_query(types, [0], AGGS, [k, v, s]))


@pytest.mark.parametrize("groups", [1, 20, 30, 1000, 3000, 60_000])
@pytest.mark.parametrize("filtered", [False, True])
def test_double_ops_and_null_keys(groups, filtered):
    """DOUBLE SUM / AVG / MIN / MAX beside counts, with NULL keys and values
    and the INT64_MIN key, in shared and HBM tables and through the warp's key
    match."""
    n = 60_011 + groups
    rng = np.random.default_rng(groups)
    k = rng.integers(0, groups, n)
    k[::977] = np.iinfo(np.int64).min
    x = rng.normal(100, 25, n)
    f = rng.integers(0, 1000, n).astype(np.int16)
    nulls = [rng.random(n) < 0.1, rng.random(n) < 0.07, None]
    types = [BIGINT, capi.DOUBLE, SMALLINT]
    aggs = [("count_star", -1), ("sum", 1), ("avg", 1), ("min", 1), ("max", 1)]
    filters = [(2, "<", 700)] if filtered else []
    cols = [k, x, f]
    orc = oracle.run_query(types, [0], aggs, cols, filters=filters, nulls=nulls)
    for options in (None, {"precombine": 1}):
        compare(run(types, [0], aggs, cols, groups, filters=filters, nulls=nulls, options=options), orc)
