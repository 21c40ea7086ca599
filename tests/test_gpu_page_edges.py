"""Compressed pages around the sizes where the page decoders change what they
do: an output window (16,384 bytes), the ring of latest output (32,768), a
parsed piece (8,192 compressed bytes), literals past what a jump holds (64 KB),
lengths that are no multiple of four; thousands of small pages (decoded by a
warp each) alone and beside large ones; ZSTD frames that the block decoder
leaves to the serial one.  Every byte reaches a group of its row number modulo
1009: exact against the oracle.  Damaged pages are refused on every path."""
import struct

import numpy as np
import pytest

import oracle
from slothdb_gb300 import capi
from slothdb_gb300 import parquet as pq
from slothdb_gb300.capi import BIGINT, INTEGER
from util import compare, gpu_to_dict

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_lib", "gblib")]

AGGS = [("sum", 1), ("min", 1), ("max", 1), ("count_star", -1)]


def ingest(data, types, devices=(False, True), options=None, profile=None):
    out = []
    for device in devices:
        pf = capi.ParquetFile(data)
        if device:
            pf.upload()
        g = capi.GroupBy(types, [0], AGGS, est_groups=1009, options=options)
        try:
            g.set_profiling(profile is not None)
            capi.ingest_parquet(g, pf, [0, 1], device=device)
            g.finalize()
            if profile is not None:
                profile.append(g.profile())
            out.append(gpu_to_dict(g.result(), 1, [INTEGER, BIGINT, types[1], types[1], BIGINT]))
        finally:
            g.close()
            pf.close()
    return out


def check(data, k, v, types=(INTEGER, BIGINT), **kw):
    types = list(types)
    orc = oracle.run_query(types, [0], AGGS, [k, v])
    for got in ingest(data, types, **kw):
        compare(got, orc)


def keys(n):
    return (np.arange(n) % 1009).astype(np.int32)


def plain(n, v, ptype=pq.T_INT64, page_rows=None, **kw):
    return pq.write([pq.Column("k", pq.T_INT32, values=keys(n)), pq.Column("v", ptype, values=v)],
                    page_rows=page_rows or n, **kw)


def pattern(kind, n, rng):
    return {"random": lambda: rng.integers(-2**31, 2**31 - 1, n), "zeros": lambda: np.zeros(n),
            "small": lambda: rng.integers(0, 300, n), "steps": lambda: np.repeat(rng.integers(0, 2**30, n // 50 + 1), 50)[:n],
            "far": lambda: np.resize(rng.integers(0, 2**30, 8189), n)}[kind]().astype(np.int32)


@pytest.mark.parametrize("n", [2040, 2045, 2046, 2047, 2048, 2049, 2050, 4095, 4096, 4097, 8191, 8192, 8193, 12_289, 16_385])
@pytest.mark.parametrize("codec", ["snappy", "zstd"])
def test_pages_around_windows(codec, n):
    rng = np.random.default_rng(n)
    for kind in ("random", "zeros", "small", "steps", "far"):
        v = pattern(kind, n, rng)
        check(plain(n, v, pq.T_INT32, codec=codec), keys(n), v, (INTEGER, INTEGER))


@pytest.mark.parametrize("codec", ["snappy", "zstd"])
def test_lengths_of_no_whole_word(codec):
    """Pages of dictionary indices: a byte a row and a few headers."""
    rng = np.random.default_rng(8)
    d = rng.permutation(1 << 20)[:256]
    for n in (1, 2, 9, 509, 1021, 8100, 8173, 16_291, 16_330, 16_373, 16_380, 32_641, 32_707, 32_767):
        for idx in (rng.integers(0, 256, n), np.arange(n) // 3 % 256):
            v = d[idx].astype(np.int64)
            data = pq.write([pq.Column("k", pq.T_INT32, values=keys(n)),
                             pq.Column("v", pq.T_INT64, dictionary=d, indices=idx.astype(np.uint32))], page_rows=n,
                            codec=codec)
            check(data, keys(n), v)


# ------------------------------------------------------------ SNAPPY elements
LITERALS = [1, 2, 59, 60, 61, 62, 63, 64, 65, 255, 256, 257, 8185, 8190, 8191, 8192, 8193, 8194, 16_383, 16_385, 57_340,
            65_500, 65_533, 65_535, 65_536, 65_537, 65_601, 70_000]


def literal(b, extra=0):
    n = len(b) - 1
    nb = 0 if n < 60 and not extra else max(1, (n.bit_length() + 7) // 8)
    nb = min(4, nb + max(0, extra - 1)) if nb else 0
    return (bytes([n << 2]) if not nb else bytes([(59 + nb) << 2]) + n.to_bytes(4, "little")[:nb]) + b


def copy(off, n, form):
    if form == 1 and 4 <= n <= 11 and off < 2048:
        return bytes([1 | ((n - 4) << 2) | ((off >> 8) << 5), off & 255])
    if form <= 2 and off < 65536:
        return bytes([2 | ((n - 1) << 2)]) + off.to_bytes(2, "little")
    return bytes([3 | ((n - 1) << 2)]) + off.to_bytes(4, "little")


def varint(n):
    out = b""
    while n >= 128:
        out += bytes([n & 127 | 128])
        n >>= 7
    return out + bytes([n])


def block(lits, rng, copies):
    """(bytes, Snappy block): the literals in turn, `copies` copies behind each."""
    raw, comp = bytearray(), bytearray()

    def lit(n):
        b = rng.integers(0, 256, n, dtype=np.uint8).tobytes()
        raw.extend(b)
        comp.extend(literal(b, int(rng.integers(0, 4))))

    for n in lits:
        lit(n)
        for _ in range(copies):
            m, off = int(rng.integers(1, 65)), int(min(len(raw), rng.choice([1, 2, 3, 5, 63, 64, 900, 2047, 30_000, 80_000])))
            comp.extend(copy(off, m, int(rng.integers(1, 5))))
            for _ in range(m):
                raw.append(raw[-off])
    if len(raw) % 8:
        lit(8 - len(raw) % 8)
    return bytes(raw), varint(len(raw)) + bytes(comp)


def with_pages(monkeypatch, name, pages):
    """The writer's compressor, but `pages` (raw -> compressed) as given."""
    real = getattr(pq, name)
    monkeypatch.setattr(pq, name, lambda data: pages.get(data) or real(data))


@pytest.mark.parametrize("first", LITERALS)
def test_snappy_literals_and_copies(monkeypatch, first):
    rng = np.random.default_rng(first)
    for lits, copies in (([first], 0), ([first, 5], 3), ([7, first, 60, first], 1), ([3] * 40 + [first] + [2] * 2000, 2)):
        raw, comp = block(lits, rng, copies)
        v = np.frombuffer(raw, "<i8")
        with monkeypatch.context() as m:
            with_pages(m, "snappy_compress", {raw: comp})
            data = plain(len(v), v, codec="snappy")
        # extreme values: MIN and MAX only are exact in the oracle's doubles
        for got in ingest(data, [INTEGER, BIGINT]):
            order = np.argsort(got["keys"][0])
            k = keys(len(v))
            for g in range(min(1009, len(v))):
                assert got["aggs"][1][0][order[g]] == v[k == g].min() and got["aggs"][2][0][order[g]] == v[k == g].max()


# ------------------------------------------------------------ many small pages
@pytest.mark.parametrize("codec", ["snappy", "zstd"])
@pytest.mark.parametrize("rows,v_rows", [(100, None), (510, None), (1030, None), (100, 40_000), (50_000, 100)])
def test_many_small_pages(codec, rows, v_rows):
    n = 430_007
    rng = np.random.default_rng(rows)
    v = np.where(rng.random(n) < 0.5, rng.integers(0, 2**40, n), 77)
    idx = rng.integers(0, 1009, n)
    data = pq.write([pq.Column("k", pq.T_INT32, dictionary=np.arange(1009, dtype=np.int32), indices=idx.astype(np.uint32)),
                     pq.Column("v", pq.T_INT64, values=v, page_rows=v_rows)], page_rows=rows, row_group_rows=200_000,
                    codec=codec)
    check(data, idx.astype(np.int32), v)


DAMAGE = {
    "far_copy": varint(800) + literal(b"x" * 8) + copy(9, 64, 2) * 13,
    "no_offset": varint(800) + literal(b"x" * 8) + copy(0, 64, 2) * 13,
    "long_literal": varint(800) + bytes([61 << 2, 0x1f, 0x03]) + b"x" * 700,
    "short": varint(800) + literal(b"x" * 8),
    "length": varint(801) + literal(b"x" * 801),
}


@pytest.mark.parametrize("damage", sorted(DAMAGE))
@pytest.mark.parametrize("pages", [1, 3000])
def test_damaged_snappy_page_is_refused(monkeypatch, damage, pages):
    n = 100 * pages
    v = np.arange(n, dtype=np.int64) % 97
    v[(n // 200) * 100:(n // 200) * 100 + 100] = 10**9 + np.arange(100)
    bad = v[(n // 200) * 100:(n // 200) * 100 + 100].astype("<i8").tobytes()
    with_pages(monkeypatch, "snappy_compress", {bad: DAMAGE[damage]})
    with pytest.raises(capi.GbError):
        ingest(plain(n, v, page_rows=100, codec="snappy"), [INTEGER, BIGINT], devices=(True,))


# ------------------------------------------------------------ unusual ZSTD frames
def raw_blocks(data, size):
    out = struct.pack("<IBI", 0xFD2FB528, 0xA0, len(data))
    for i in range(0, len(data), size):
        part = data[i:i + size]
        out += struct.pack("<I", (i + size >= len(data)) | len(part) << 3)[:3] + part
    return out


def rle_frame(byte, n):
    return struct.pack("<IBI", 0xFD2FB528, 0xA0, n) + struct.pack("<I", 1 | 1 << 1 | n << 3)[:3] + byte


def odd_frames(real, every, form):
    count = [0]

    def compress(data):
        count[0] += 1
        if count[0] % every or len(data) < 16:
            return real(data)
        q = len(data) // 3
        if form == "frames":
            return real(data[:q]) + real(data[q:2 * q]) + real(data[2 * q:])
        if form == "skippable":
            return struct.pack("<II", 0x184D2A53, 5) + b"hello" + real(data)
        return raw_blocks(data, 200)  # more blocks than descriptors

    return compress


@pytest.mark.parametrize("form", ["frames", "skippable", "blocks"])
@pytest.mark.parametrize("every,rows", [(1, 4000), (3, 4000), (2, 50_000), (1, 150)])
def test_odd_zstd_frames_beside_regular_ones(monkeypatch, form, every, rows):
    n = 300_001
    rng = np.random.default_rng(every + rows)
    v = np.where(rng.random(n) < 0.6, rng.integers(0, 5000, n), 2**39)
    monkeypatch.setattr(pq, "zstd_compress", odd_frames(pq.zstd_compress, every, form))
    check(plain(n, v, page_rows=rows, codec="zstd"), keys(n), v)


def test_raw_and_run_length_blocks(monkeypatch):
    n = 40_000
    v = np.zeros(n, np.int64)
    v[100:200] = np.arange(100)
    pages = {v[:20_000].tobytes(): raw_blocks(v[:20_000].tobytes(), 100_000),
             v[20_000:].tobytes(): rle_frame(b"\0", 160_000)}
    with_pages(monkeypatch, "zstd_compress", pages)
    check(plain(n, v, page_rows=20_000, codec="zstd"), keys(n), v)


# ------------------------------------------------------------ times
def kernel_ms(data, prefix):
    best = None
    for _ in range(4):
        p = []
        ingest(data, [INTEGER, BIGINT], devices=(True,), profile=p)
        ms = sum(t[1] for k, t in p[0].items() if k.startswith(prefix))
        best = ms if best is None else min(best, ms)
    return best


def test_small_pages_cost_no_more_than_large_ones():
    """The same rows in pages of 200 and of 8,192 rows: a block for each small
    page took 10 times as long as the large ones, a warp a fraction."""
    n = 400_000
    v = np.random.default_rng(1).integers(0, 10**6, n)
    small, large = (kernel_ms(plain(n, v, page_rows=r, codec="snappy"), "k_pq_inflate") for r in (200, 8192))
    assert small <= 2 * large, (small, large)


def test_odd_pages_use_the_whole_gpu(monkeypatch):
    """4,800 pages of three frames against 600 of them: with four decoding
    warps an SM they took 8 rounds to one, with twenty 2."""
    monkeypatch.setattr(pq, "zstd_compress", odd_frames(pq.zstd_compress, 1, "frames"))
    rng = np.random.default_rng(2)
    ms = []
    for pages in (600, 4800):
        v = rng.integers(0, 10**6, 500 * pages // 2)
        ms.append(kernel_ms(plain(len(v), v, page_rows=500, codec="zstd"), "k_pz_"))
    assert ms[1] <= 4 * ms[0], ms


@pytest.mark.parametrize("scratch", [0, 40 << 20, 9 << 20, 1_300_000, 100_000, 1])
def test_zstd_scratch_that_is_short(scratch):
    """24 pages of up to 200 KB: in one group, in several, in one for each page,
    and with no scratch at all by the serial decoder."""
    n = 300_000
    rng = np.random.default_rng(6)
    v = np.where(rng.random(n) < 0.6, rng.integers(0, 5000, n), 2**39)
    prof = []
    check(plain(n, v, page_rows=25_000, codec="zstd"), keys(n), v, options={"zstd_scratch": scratch}, profile=prof)
    for p in prof:
        groups = p["k_pz_blocks"][0]
        if scratch == 0:
            assert groups == 1 and p["k_pz_entropy"][0] == 1
        elif scratch < 10**6:
            assert groups == 1 and "k_pz_entropy" not in p
        else:
            assert groups == p["k_pz_entropy"][0] and (groups > 1) == (scratch < 20 << 20)
