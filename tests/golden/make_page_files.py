"""Parquet files whose compressed pages are large (written by pyarrow's SNAPPY
and ZSTD) for the page decoders' parity tests — regenerated by running this
script from the repository root:  python tests/golden/make_page_files.py

The GPU machine has no pyarrow, so the files are committed (gzipped); their
logical columns are regenerated by `columns()` (numpy only).  The ZSTD pages
hold frames of several blocks with Huffman literals (own and earlier tables),
described, predefined, repeated and one-symbol sequence tables and repeat
offsets that reach over block boundaries; the SNAPPY pages hold its encoder's
64 KB fragments.
"""
from __future__ import annotations

import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from make_pyarrow_files import _write  # noqa: E402

FILES = {"pa_pages_zstd1": ("zstd", 1), "pa_pages_zstd9": ("zstd", 9), "pa_pages_zstd19": ("zstd", 19),
         "pa_pages_snappy": ("snappy", None)}
N = 72_000


def columns(n=N, seed=41):
    """k INT32 (row number modulo 1009) and v INT64 in stretches of other byte statistics."""
    rng = np.random.default_rng(seed)
    m = n // 6
    words = [b"alpha   ", b"beta    ", b"gamma-01", b"delta-22", b"epsilon "]
    v = np.concatenate([
        np.cumsum(rng.integers(0, 3, m)),                                               # slow growth
        np.frombuffer(b"".join(words[i] for i in rng.integers(0, 5, m)), dtype="<i8") >> 20,  # words
        np.zeros(m, dtype=np.int64),                                                    # one long run
        np.tile(rng.integers(0, 2**40, 97), m // 97 + 1)[:m],                           # a period of 776 bytes
        rng.integers(0, 1000, m),                                                       # small values
        rng.integers(-2**20, 2**20, m)])                                                # wider ones
    v = np.concatenate([v, np.arange(n - len(v))]).astype(np.int64)
    return (np.arange(n) % 1009).astype(np.int32), v


def main():
    import pyarrow as pa
    k, v = columns()
    t = pa.table([pa.array(k), pa.array(v)], schema=pa.schema([pa.field("k", pa.int32(), nullable=False),
                                                               pa.field("v", pa.int64(), nullable=False)]))
    for name, (codec, level) in FILES.items():
        _write(name, t, compression=codec, compression_level=level, row_group_size=N, data_page_size=8 << 20,
               use_dictionary=False)


if __name__ == "__main__":
    main()
