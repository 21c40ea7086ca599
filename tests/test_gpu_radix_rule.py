"""The table size of the radix pipeline's DOUBLE sums where the partitions are
fewer than the estimate asks for (keys that take the generic partition pass, a
set partition count) or the estimate is too low: groups that fit the tables
must not go through the HBM table, whose growth would be launches of its own;
results exact (counts) and within the oracle tests' relative tolerance."""
import numpy as np
import pytest

import oracle
from slothdb_gb300 import capi
from slothdb_gb300.capi import BIGINT, DOUBLE, INTEGER
from util import compare, gpu_to_dict

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_lib", "gblib")]

AGGS = [("count_star", -1), ("sum", 1), ("avg", 1)]


def run(key_type, k, x, est, bits=None):
    options = {"mode": 2}
    if bits:
        options["radix_bits"] = bits
    g = capi.GroupBy([key_type, DOUBLE], [0], AGGS, est_groups=est, options=options)
    try:
        g.ingest([k, x], nrows=len(k))
        g.finalize()
        return g.result(), g.launches()
    finally:
        g.close()


# est: what the generic pass's 1,024 partitions of small tables hold is passed
# at 7.3M; 100,000 is far below the 400,000 groups that come
@pytest.mark.parametrize("key_type,groups,est,bits", [
    (INTEGER, 7_200_000, 7_200_000, None), (INTEGER, 7_400_000, 7_400_000, None), (INTEGER, 11_500_000, 11_500_000, None),
    (BIGINT, 400_000, 100_000, None), (BIGINT, 700_000, 700_000, 6), (INTEGER, 700_000, 700_000, 6)])
def test_groups_that_fit_stay_in_the_tables(key_type, groups, est, bits):
    rng = np.random.default_rng(groups)
    k = np.arange(groups, dtype=np.int64)
    rng.shuffle(k)
    k = k.astype(np.int32) if key_type == INTEGER else k * 1_000_003
    x = rng.normal(100, 25, groups)
    res, launches = run(key_type, k, x, est, bits)
    _, few = run(key_type, k[:5000], x[:5000], est, bits)
    assert launches == few  # nothing spilled: no rehash, no merge
    order = np.argsort(res[0][0])
    np.testing.assert_array_equal(res[0][0][order], np.sort(k))
    assert (res[1][0] == 1).all()  # each group is one row: its sum and average are the value
    at = np.argsort(k)
    np.testing.assert_array_equal(res[2][0][order], x[at])
    np.testing.assert_array_equal(res[3][0][order], x[at])


@pytest.mark.parametrize("key_type", [BIGINT, INTEGER])
@pytest.mark.parametrize("bits", [None, 6])
def test_tables_that_overflow(key_type, bits):
    """Four and more groups for every slot of the tables."""
    rng = np.random.default_rng(3)
    n, groups = 5_000_000, 4_500_000
    k = rng.integers(0, groups, n)
    k = k.astype(np.int32) if key_type == INTEGER else k * 1_000_003
    x = rng.normal(100, 25, n)
    res, _ = run(key_type, k, x, 100_000, bits)
    compare(gpu_to_dict(res, 1, [key_type, BIGINT, DOUBLE, DOUBLE]),
            oracle.run_query([key_type, DOUBLE], [0], AGGS, [k, x]))
