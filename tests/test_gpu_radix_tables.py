"""The radix pipeline's DOUBLE-sum tables on both sides of the estimate where
their size changes, empty and full partitions and CTAs of several partitions;
the register TopN against the general one."""
import numpy as np
import pytest

import oracle
from slothdb_gb300 import capi
from slothdb_gb300.capi import BIGINT, DOUBLE, SMALLINT
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


@pytest.mark.parametrize("limit", [1, 2, 10, 15, 16, 17, 31, 32])
@pytest.mark.parametrize("groups", [1, 9, 33, 4097, 200_000])
def test_topn_lists_equal_the_general_path(limit, groups):
    """Ties in the order column, NULLs among it, both directions, every type."""
    rng = np.random.default_rng(groups + limit)
    n = 2 * groups + 77
    k = (rng.integers(0, groups, n) - groups // 2).astype(np.int64)
    v = rng.integers(-40, 40, n)
    x = np.round(rng.normal(0, 3, n))
    s = rng.integers(-9, 9, n).astype(np.int16)
    types = [BIGINT, BIGINT, DOUBLE, SMALLINT]
    aggs = [("count_star", -1), ("sum", 1), ("max", 2), ("min", 3)]
    nulls = [None, rng.random(n) < 0.4, rng.random(n) < 0.4, rng.random(n) < 0.4]
    for col in range(1, 5):
        for ascending in (False, True):
            a, b = (result(types, [0], aggs, [k, v, x, s], groups, topn=(col, ascending, limit), nulls=nulls,
                           options={"topn_small": small}) for small in (1, 0))
            assert len(a) == len(b)
            for p, q in zip(a, b):
                for u, w in zip(p, q):
                    np.testing.assert_array_equal(np.asarray(u), np.asarray(w))
