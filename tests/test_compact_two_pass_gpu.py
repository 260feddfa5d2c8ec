"""GPU parity of the NULL split and of the two-pass row-id compaction (run starts, unaligned columns), around the
size the two-pass form starts at and at the edges of their tiles and scan groups, against numpy, exactly."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import bitmap

pytestmark = pytest.mark.gpu

ROWS = 1 << 20  # the two-pass form starts here; 2,048-row tiles, 4,096 tiles a scan group
SIZES = [ROWS - 1, ROWS, ROWS + 1, ROWS + 2048 * 3 + 7, 2048 * 4096 - 1, 2048 * 4096, 2048 * 4096 + 1, 2048 * 16_384 + 2049]


@pytest.mark.parametrize("nulls_first", [False, True])
@pytest.mark.parametrize("n", SIZES)
def test_null_split(bolt, engine, n, nulls_first):
    """Two keys: the second split reads its rows through the first's order (ids_in)."""
    rng = np.random.default_rng(n)
    a, b = rng.integers(0, 3, n).astype(np.int32), rng.integers(-9, 9, n).astype(np.int32)
    va, vb = rng.random(n) > 0.3, rng.random(n) > 0.6
    cols = [bolt.col(a, "i32", bitmap(va)).to("cuda"), bolt.col(b, "i32", bitmap(vb)).to("cuda")]
    got = engine.sort_indices(cols, False, nulls_first).cpu().numpy().view(np.uint32)
    s = 1 if nulls_first else -1
    want = np.lexsort((np.where(vb, b, 0), s * vb.astype(np.int8), np.where(va, a, 0), s * va.astype(np.int8)))
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n", SIZES[:4])
@pytest.mark.parametrize("keep", [0, 3, 100])
def test_unaligned_columns(bolt, engine, n, keep):
    """Columns off a 16-byte boundary with a validity bitmap take the direct kernel, rows and bits alike."""
    rng = np.random.default_rng(n + keep)
    buf = torch.from_numpy(rng.integers(0, 100, n + 3).astype(np.int32)).cuda()
    f, wide = buf[1:n + 1], torch.arange(n + 1, dtype=torch.int64, device="cuda")[1:]
    valid = rng.random(n) > 0.2
    t = {"f": bolt.col(f), "x": bolt.Column(wide, "i64", torch.from_numpy(bitmap(valid)).cuda())}
    cols, rid = engine.compact_columns(t, where=[("f", "<", keep)])
    m = f.cpu().numpy() < keep
    assert np.array_equal(rid.cpu().numpy(), np.flatnonzero(m))
    assert np.array_equal(cols["x"].numpy(), np.flatnonzero(m) + 1)
    assert np.array_equal(cols["x"].valid_mask(), valid[m])
