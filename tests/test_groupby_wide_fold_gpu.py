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


def _lengths(n_groups, long_at):
    """1 or 2 rows a group, but for the groups of long_at: {group: rows}."""
    lengths = 1 + np.arange(n_groups) % 2
    for g, rows in long_at.items():
        lengths[g] = rows
    return lengths


def _by_length(bolt, oracle, rng, lengths):
    group = rng.permutation(np.repeat(np.arange(len(lengths)), lengths))
    cols = _columns(rng, len(group), ("i64", "i32"), 1, key_nulls=False)
    cols["k0"] = ((group >> 4).astype(np.int64) * (1 << 35) - 5, None, "i64")
    cols["k1"] = ((group & 15).astype(np.int32), None, "i32")
    return _tables(bolt, oracle, cols)


def test_long_groups_among_many(bolt, engine, oracle):
    """More groups than 32 a warp of the grid (148 SMs x 64 warps): long ones next to each other, at the ends of the
    grid's rounds (9,472 warps) and of 32 rounds (303,104 groups), and the very last."""
    n_groups = 350_011
    warps = 148 * 64
    long_at = {g: 49 + 251 * i // 40 for i, g in enumerate(
        [0, 1, 2, 31, 32, 33, 63, 64, warps - 1, warps, warps + 1, 2 * warps, 31 * warps - 1, 31 * warps, 32 * warps - 2,
         32 * warps - 1, 32 * warps, 32 * warps + 1, 33 * warps] + list(range(200_000, 200_016)) + [n_groups - 2, n_groups - 1])}
    rng = np.random.default_rng(2)
    dev, host = _by_length(bolt, oracle, rng, _lengths(n_groups, long_at))
    res = engine.execute_groupby(dev, ["k0", "k1"], AGGS)
    assert res.n_groups == n_groups
    _check(res, oracle.groupby_wide(host, ["k0", "k1"], AGGS), AGGS)


def test_long_neighbours_fold_side_by_side(bolt, engine, oracle):
    """Sixteen long groups next to each other in key order, among more groups than 32 a warp: their folds are chains
    of dependent adds and must not follow one another, so together they take little more than one of them."""
    n_groups, rows = 350_011, 60_000
    ms = []
    for long_at in ({200_000: rows}, {200_000 + i: rows for i in range(16)}):
        dev, _ = _by_length(bolt, oracle, np.random.default_rng(3), _lengths(n_groups, long_at))
        least = []
        for _ in range(3):
            assert engine.execute_groupby(dev, ["k0", "k1"], [("sum", "vd")], groups_hint=n_groups).n_groups == n_groups
            least.append(engine.last_device_ms)
        ms.append(min(least))
    assert ms[1] <= 3 * ms[0]


@pytest.mark.parametrize("n_groups", [9_471, 9_472, 9_473, 18_944, 18_945, 28_417])
def test_hand_over_by_group_count(bolt, engine, oracle, n_groups):
    """The length from which a warp folds a group rises with the groups per warp of the chip (148 x 64): 8, 24, 40,
    48 rows. Groups of every length around them, in one query."""
    edges = np.array([1, 2, 7, 8, 9, 23, 24, 25, 39, 40, 41, 47, 48, 49, 60])
    lengths = np.where(np.arange(n_groups) % 19 == 0, edges[np.arange(n_groups) // 19 % len(edges)], 2)
    rng = np.random.default_rng(n_groups)
    dev, host = _by_length(bolt, oracle, rng, lengths)
    res = engine.execute_groupby(dev, ["k0", "k1"], AGGS)
    assert res.n_groups == n_groups
    _check(res, oracle.groupby_wide(host, ["k0", "k1"], AGGS), AGGS)


def test_few_short_groups_cost_no_more_than_longer_ones(bolt, engine, oracle):
    """A thousand groups, every aggregate: 48 rows each against 49, which warps fold."""
    ms = []
    for rows in (48, 49):
        dev, _ = _by_length(bolt, oracle, np.random.default_rng(4), np.full(1000, rows))
        least = []
        for _ in range(9):
            engine.execute_groupby(dev, ["k0", "k1"], AGGS, groups_hint=1000)
            least.append(engine.last_device_ms)
        ms.append(min(least))
    print(f"48 rows {ms[0] * 1e3:.1f} us, 49 rows {ms[1] * 1e3:.1f}")
    assert ms[0] <= 1.1 * ms[1]
