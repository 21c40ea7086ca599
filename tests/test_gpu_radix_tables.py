"""The radix pipeline's DOUBLE-sum tables on both sides of the estimate where
their size changes, empty and full partitions and CTAs of several partitions."""
import numpy as np
import pytest

import oracle
from slothdb_gb300 import capi
from slothdb_gb300.capi import BIGINT, DOUBLE
from util import compare, gpu_to_dict

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_lib", "gblib")]


def result(types, keys, aggs, cols, est, topn=None, options=None, nulls=None, runs=1):
    words = None
    nullable = []
    if nulls is not None:
        words = [None if m is None else capi.validity_words(~m) for m in nulls]
        nullable = [i for i, m in enumerate(nulls) if m is not None]
    g = capi.GroupBy(types, keys, aggs, est_groups=est, nullable=nullable, options=options)
    try:
        if topn:
            g.set_topn(*topn)
        for _ in range(runs):
            g.reset()
            g.ingest(cols, nrows=len(cols[0]), validity=words)
            g.finalize()
        return g.result()
    finally:
        g.close()


@pytest.mark.parametrize("est", [1 << 20, 23_400_000, 23_600_000, 50_000_000])
@pytest.mark.parametrize("groups", [1, 700, 90_000, 1_500_000])
def test_double_sum_tables(est, groups):
    rng = np.random.default_rng(groups)
    n = groups + 400_003
    k = rng.permutation(np.arange(n) % groups) * 1_640_531_527 % (1 << 40)
    k[5::1009] = np.iinfo(np.int64).min
    x = rng.normal(100, 25, n)
    types, aggs = [BIGINT, DOUBLE], [("count_star", -1), ("avg", 1), ("count", 1), ("sum", 1)]
    out = [BIGINT] + [oracle.agg_out_type(oracle.AGG_NAMES[a], types[c] if c >= 0 else 0) for a, c in aggs]
    got = gpu_to_dict(result(types, [0], aggs, [k, x], est, runs=2), 1, out)
    compare(got, oracle.run_query(types, [0], aggs, [k, x]))

