"""Growth of the HBM table with keys whose hashes agree in their low bits, so
that their probe runs are longer than the probe bound (256) in every capacity
up to 2^14: the rehash spills records of its own behind those that are pending,
more of them than pending ones; nothing may be lost or counted twice."""
import numpy as np
import pytest

from slothdb_gb300 import capi
from slothdb_gb300.capi import BIGINT

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("gblib")]

LOW = 14


def mix64(k):
    k = k.astype(np.uint64)
    k ^= k >> np.uint64(33)
    k *= np.uint64(0xff51afd7ed558ccd)
    k ^= k >> np.uint64(33)
    k *= np.uint64(0xc4ceb9fe1a85ec53)
    return k ^ (k >> np.uint64(33))


@pytest.fixture(scope="module")
def homes():
    k = np.arange(1, 1 << 23, dtype=np.int64)
    return k, (mix64(k) & np.uint64((1 << LOW) - 1)).astype(np.int64)


@pytest.mark.parametrize("home", [100, 1000])
@pytest.mark.parametrize("first,second,apart", [(160, 160, 60), (200, 200, 100), (230, 230, 200), (250, 20, 5)])
def test_rehash_that_spills(homes, home, first, second, apart):
    k, h = homes
    a, b = k[h == home][:first], k[h == home + apart][:second]
    assert len(a) == first and len(b) == second
    rng = np.random.default_rng(first)
    parts = [np.repeat(a, 3), np.repeat(b, 2), rng.permutation(np.concatenate([a, b]))]
    vals = [rng.integers(-10**9, 10**9, len(p)) for p in parts]
    want = {}
    for p, v in zip(parts, vals):
        for x, y in zip(p.tolist(), v.tolist()):
            c, s, m = want.get(x, (0, 0, y))
            want[x] = (c + 1, s + y, min(m, y))
    for _ in range(5):  # the order of a parallel rehash varies
        g = capi.GroupBy([BIGINT, BIGINT], [0], [("count_star", -1), ("sum", 1), ("min", 1)], est_groups=1,
                         options={"mode": 1})
        try:
            for p, v in zip(parts, vals):
                g.ingest([p, v])
            g.finalize()
            res = g.result()
        finally:
            g.close()
        got = {x: t for x, *t in zip(*(c[0].tolist() for c in res))}
        assert len(res[0][0]) == len(got) == len(want)
        assert all(tuple(got[x]) == w for x, w in want.items())
