"""ORDER BY within the scratch it has always needed, and no more: two key and row buffers, the look-back words of the
tiles and the digit tables."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import bitmap

pytestmark = pytest.mark.gpu

N = 4_000_003
TABLES = 2 * 8 * 256 * 4 + 8192  # digit tables; ten buffers rounded up to 256 bytes, counters


@pytest.mark.parametrize("dt,width,tile", [(np.int64, 8, 4096), (np.int32, 4, 5120)])
def test_one_key(bolt, dt, width, tile):
    v = np.random.default_rng(width).integers(np.iinfo(dt).min, np.iinfo(dt).max, N, dtype=dt)
    engine = bolt.Engine(0, scratch_bytes=2 * N * (width + 4) + 2 * 256 * 4 * -(-N // tile) + TABLES)
    try:
        got = engine.sort_indices([bolt.col(v).to("cuda")]).cpu().numpy().view(np.uint32)
    finally:
        engine.close()
    assert np.array_equal(got, np.argsort(v, kind="stable"))


# Room for the valid rows' ids, and eight bytes twice for every 2,048 rows; 64 rows sort in 64 KB.
@pytest.mark.parametrize("valid_rows", [0, 64])
@pytest.mark.parametrize("nulls_first", [False, True])
def test_nulls(bolt, valid_rows, nulls_first):
    """A column of hardly more than NULLs needs little beside its valid rows' ids."""
    rng = np.random.default_rng(valid_rows)
    v = rng.integers(-9, 9, N)
    valid = np.zeros(N, bool)
    valid[rng.permutation(N)[:valid_rows]] = True
    engine = bolt.Engine(0, scratch_bytes=4 * N + 16 * (N // 2048 + 2) + (65_536 if valid_rows else 2048))
    try:
        got = engine.sort_indices([bolt.col(v, "i64", bitmap(valid)).to("cuda")], False, nulls_first)
    finally:
        engine.close()
    nulls, rest = np.flatnonzero(~valid), np.flatnonzero(valid)
    rest = rest[np.argsort(v[rest], kind="stable")]
    want = np.concatenate([nulls, rest] if nulls_first else [rest, nulls])
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want)


def test_nulls_of_two_keys(bolt):
    """The same behind another key, so that the split reads its rows through an order."""
    rng = np.random.default_rng(3)
    a, b = rng.integers(-9, 9, N), rng.integers(0, 4, N)
    valid = np.zeros(N, bool)
    valid[rng.permutation(N)[:1000]] = True
    need = max(2 * N * 12 + 2 * 256 * 4 * -(-N // 4096) + TABLES, 4 * N + 16 * (N // 2048 + 2) + 65_536)
    engine = bolt.Engine(0, scratch_bytes=4 * N + 256 + need)
    try:
        got = engine.sort_indices([bolt.col(a, "i64", bitmap(valid)).to("cuda"), bolt.col(b).to("cuda")])
    finally:
        engine.close()
    want = np.lexsort((b, np.where(valid, a, 0), ~valid))
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want)
