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
