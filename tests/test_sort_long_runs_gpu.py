"""Runs of equal top digits longer than the local step's window, mostly one value among others of its run: the order
against numpy's stable argsort, and the time against keys for which every digit gets a pass."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _full(rng, n):
    return rng.integers(-(1 << 63), (1 << 63) - 1, n, dtype=np.int64)


def _sort(bolt, engine, v, reps=1):
    """(permutation, least device time in ms)"""
    col = bolt.col(v).to("cuda")
    ms = []
    for _ in range(reps):
        perm = engine.sort_indices([col])
        ms.append(engine.last_device_ms)
    return perm.cpu().numpy().view(np.uint32), min(ms)


def _hot(rng, n, hot, others):
    """Uniform keys, of which `hot` are 0 and `others` are ids that share its top three bytes."""
    v = _full(rng, n)
    at = rng.permutation(n)
    v[at[:hot]] = 0
    v[at[hot:hot + others]] = rng.integers(1, 1 << 40, others)
    return v


# 5,120 rows of other values: one window of 64-bit keys.
@pytest.mark.parametrize("others", [5119, 5120, 5121, 8000])
@pytest.mark.parametrize("n,hot", [(3_000_017, 40_000), (1 << 24, 200_001)])
def test_others_around_one_window(bolt, engine, n, hot, others):
    v = _hot(np.random.default_rng(others), n, hot, others)
    got, _ = _sort(bolt, engine, v)
    assert np.array_equal(got, np.argsort(v, kind="stable"))


def test_no_slower_than_every_digit(bolt, engine):
    """2^24 keys, 1.2 % of one value and 8,000 ids beside it, against keys that crowd (one pass per digit). The bound
    is the schedule's purpose: it is taken to be faster than the passes it leaves out."""
    n = 1 << 24
    rng = np.random.default_rng(1)
    v = _hot(rng, n, 200_000, 8_000)
    got, ms = _sort(bolt, engine, v, 5)
    assert np.array_equal(got, np.argsort(v, kind="stable"))
    crowded = _full(rng, n)
    crowded[::2] = (crowded[::2] & 0xFFFFFFFFFF) + (5 << 40)
    got, all_ms = _sort(bolt, engine, crowded, 5)
    assert np.array_equal(got, np.argsort(crowded, kind="stable"))
    assert ms <= all_ms


def test_crowded_window_costs_little(bolt, engine):
    """One window whose keys crowd into a few bins, against uniform keys: a crowded chunk is one block's work, and the
    grid ends with it."""
    n = 5000
    rng = np.random.default_rng(8)
    v = _full(rng, n)
    _, uniform_ms = _sort(bolt, engine, v, 25)
    v[::2] = (v[::2] & 0xFFFFFF) + (5 << 40)
    got, ms = _sort(bolt, engine, v, 25)
    assert np.array_equal(got, np.argsort(v, kind="stable"))
    print(f"crowded {ms * 1e3:.1f} us, uniform {uniform_ms * 1e3:.1f}")
    assert ms - uniform_ms <= 0.032  # (38 us with a counting pass per digit, 26 by merging)


# 5,120 rows: one window; 10 rows: what one thread sorts by itself.
@pytest.mark.parametrize("n", [33, 5000, 5111, 5119, 5120])
@pytest.mark.parametrize("values", [2, 90])
def test_crowded_window(bolt, engine, n, values):
    """Few values far apart and clusters around them, in one window: the bins are too long, the merge sort orders it."""
    rng = np.random.default_rng(n * values)
    v = rng.choice(_full(rng, values), n)
    near = rng.random(n) < 0.5
    v[near] ^= rng.integers(0, 64, near.sum())
    for x in (v, v >> 40, (v >> 32).astype(np.int32)):
        got, _ = _sort(bolt, engine, x)
        assert np.array_equal(got, np.argsort(x, kind="stable"))


@pytest.mark.parametrize("n", [1_000_003, 3_000_017])
@pytest.mark.parametrize("length", [8_000, 16_000])
def test_long_run_is_seen(bolt, engine, n, length):
    """A run of many values longer than a window, against keys that get a pass for every digit: the sample must see
    the run before its one block takes longer than the passes left out."""
    rng = np.random.default_rng(n + length)
    v = _full(rng, n)
    every = v.copy()
    v[rng.permutation(n)[:length]] = (0x1111111 << 32) + rng.integers(0, 1 << 32, length)
    got, ms = _sort(bolt, engine, v, 9)
    assert np.array_equal(got, np.argsort(v, kind="stable"))
    every[::2] = (every[::2] & 0xFFFF) + (5 << 40)
    got, every_ms = _sort(bolt, engine, every, 9)
    assert np.array_equal(got, np.argsort(every, kind="stable"))
    print(f"{n} rows, run of {length}: {ms * 1e3:.1f} us, every digit {every_ms * 1e3:.1f}")
    assert ms <= every_ms
