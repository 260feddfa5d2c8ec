"""Wide-key GROUP BY: groups around the length at which one thread's fold hands over to one warp's, mixed in
one query, bit for bit against the oracle (floats in row order, NULLs, NaN and signed zeros among them)."""

from __future__ import annotations

import numpy as np
import pytest

from test_groupby_wide_gpu import AGGS, _check, _columns, _tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [[48], [49], [1, 2, 3, 4, 5, 47, 48, 49, 50, 95, 96, 97, 1, 300],
                                     [7] * 100 + [48, 49] * 40 + [1] * 33])
def test_lengths_around_the_hand_over(bolt, engine, oracle, lengths):
    rng = np.random.default_rng(len(lengths))
    group = rng.permutation(np.repeat(np.arange(len(lengths)), lengths))
    cols = _columns(rng, len(group), ("i64", "i32"), 1, key_nulls=False)
    cols["k0"] = (group.astype(np.int64) * (1 << 35) - 5, None, "i64")
    cols["k1"] = ((group % 3).astype(np.int32), None, "i32")
    dev, host = _tables(bolt, oracle, cols)
    res = engine.execute_groupby(dev, ["k0", "k1"], AGGS)
    assert res.n_groups == len(lengths)
    _check(res, oracle.groupby_wide(host, ["k0", "k1"], AGGS), AGGS)
