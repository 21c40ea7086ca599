"""Ingests whose keys find no slot in the HBM table, up to every row: the spill
buffer holds a record for each row of a small ingest, and of a large one the
threshold and what the CTAs' tiles in hand still add; then the table grows and
the rest follows.  Integers exact, sums of whole-valued DOUBLEs too."""
import numpy as np
import pytest

from slothdb_gb300 import capi
from slothdb_gb300.capi import BIGINT, DOUBLE

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("gblib")]


@pytest.mark.parametrize("rows", [1_000, 40_000, 900_000, 1_100_000, 3_000_000, 7_000_000])
@pytest.mark.parametrize("types,fast", [((BIGINT, BIGINT), 1), ((BIGINT, DOUBLE), 1), ((BIGINT, BIGINT), 0)])
@pytest.mark.parametrize("options", [{}, {"smem_slots": 0}, {"ctas_per_sm": 4, "tile_rows": 512}])
def test_every_row_a_new_group(rows, types, fast, options):
    import torch
    rng = np.random.default_rng(rows)
    k = rng.permutation(rows).astype(np.int64) * 10_007 - 10**9
    v = rng.integers(-10**6, 10**6, rows)
    x = v.astype(np.float64) if types[1] == DOUBLE else v
    g = capi.GroupBy(list(types), [0], [("count_star", -1), ("sum", 1)], est_groups=16,
                     options=dict(options, mode=1, fast_ingest=fast))
    try:
        for _ in range(2):
            g.reset()
            g.ingest([torch.from_numpy(k).cuda(), torch.from_numpy(x).cuda()], nrows=rows, device=True)
            g.ingest([k[:rows // 3], x[:rows // 3]], nrows=rows // 3)  # known groups again, from host memory
            g.finalize()
        res = g.result()
    finally:
        g.close()
    assert len(res[0][0]) == rows
    order, want = np.argsort(res[0][0]), np.argsort(k)
    twice = np.arange(rows) < rows // 3
    np.testing.assert_array_equal(res[0][0][order], k[want])
    np.testing.assert_array_equal(res[1][0][order], (1 + twice)[want])
    np.testing.assert_array_equal(res[2][0][order], (v * (1 + twice))[want])
