"""GPU parity of the short sort schedule (passes over the top digits, then the local step) against numpy's
stable argsort, bit-exact: the key distributions and sizes where its work items, runs and bins have edges."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import bitmap

pytestmark = pytest.mark.gpu

M = 1_000_003


def _keys(name: str, n: int) -> np.ndarray:
    rng = np.random.default_rng(n + len(name))
    full = rng.integers(-(1 << 63), (1 << 63) - 1, n, dtype=np.int64)
    if name == "full":
        return full
    if name == "narrow":  # 40 varying bits around zero: the constant bytes get no digit
        return rng.integers(-(1 << 39), 1 << 39, n)
    if name == "packed":  # two small fields with constant bytes between them
        return (rng.integers(0, 1000, n) << 32) | rng.integers(0, 1000, n)
    if name == "long_run":  # one run of equal top bytes longer than a window, inside uniform keys
        at = rng.permutation(n)[: min(n // 2, 20_000)]
        full[at] = (np.int64(0x1234567890) << 24) | rng.integers(0, 1 << 24, len(at))
        return full
    if name == "one_value":  # the same, all keys of the run equal
        full[rng.permutation(n)[: min(n // 2, 20_000)]] = 42
        return full
    if name == "dups":  # every key about 200 times: bins too long to rank
        return rng.choice(full[: max(1, n // 200)], n)
    if name == "few":  # two varying bytes: full LSD
        return rng.integers(0, 60_000, n)
    assert name == "sorted"
    return np.sort(full)


NAMES = ["full", "narrow", "packed", "long_run", "one_value", "dups", "few", "sorted"]


# 5,120 rows: one window of the local step; 4,096 rows: its work item at these sizes, ten of them and a row.
@pytest.mark.parametrize("n", [33, 5119, 5120, 5121, 8191, 8193, 40_961, M])
@pytest.mark.parametrize("name", NAMES)
def test_i64(bolt, engine, name, n):
    v = _keys(name, n)
    got = engine.sort_indices([bolt.col(v).to("cuda")]).cpu().numpy().view(np.uint32)
    assert np.array_equal(got, np.argsort(v, kind="stable"))
    down = engine.sort_indices([bolt.col(v).to("cuda")], True).cpu().numpy().view(np.uint32)
    assert np.array_equal(down, np.argsort(~v, kind="stable"))


# 6,144 rows: one window of 32-bit keys.
@pytest.mark.parametrize("n", [6143, 6144, 6145, 100_001, M])
@pytest.mark.parametrize("name", ["full", "narrow", "long_run", "dups"])
def test_i32_and_floats(bolt, engine, name, n):
    v32 = (_keys(name, n) >> (0 if name == "dups" else 20)).astype(np.int32)
    got = engine.sort_indices([bolt.col(v32).to("cuda")]).cpu().numpy().view(np.uint32)
    assert np.array_equal(got, np.argsort(v32, kind="stable"))
    rng = np.random.default_rng(n)
    for dt in (np.float32, np.float64):
        f = (np.power(10.0, rng.random(n) * 8 - 2) * rng.choice([-1.0, 1.0], n)).astype(dt)
        f[::1001] = 0.0
        f[7::1001] = -0.0
        f[9::1001] = np.nan
        f[11::1001] = np.inf
        got = engine.sort_indices([bolt.col(f).to("cuda")]).cpu().numpy().view(np.uint32)
        assert np.array_equal(got, np.argsort(f, kind="stable"))


def test_runs_longer_than_a_window(bolt, engine):
    """Runs of equal top digits past the local step's window, few enough rows to stay on the short schedule: of
    many values, of one value among others of its run, and of one value alone."""
    n = 3_000_017
    v = _keys("full", n)
    rng = np.random.default_rng(3)
    at = rng.permutation(n)[: 9 * 8000].reshape(9, 8000)
    for i in range(3):
        v[at[i]] = (np.int64(0x1111111 * (i + 1)) << 32) | rng.integers(0, 1 << 32, 8000)
        v[at[3 + i]] = np.int64(0x2222222222 * (i + 1))
        v[at[6 + i]] = (np.int64(-0x3333333 * (i + 1)) << 32) | np.where(rng.random(8000) < 0.6, 77, rng.integers(0, 1 << 20, 8000))
    got = engine.sort_indices([bolt.col(v).to("cuda")]).cpu().numpy().view(np.uint32)
    assert np.array_equal(got, np.argsort(v, kind="stable"))
    f = rng.normal(0, 1e3, n)
    f[at[0]], f[at[1]], f[at[2]], f[at[3]] = 0.0, -0.0, np.nan, np.inf
    for x in (f, f.astype(np.float32)):
        got = engine.sort_indices([bolt.col(x).to("cuda")]).cpu().numpy().view(np.uint32)
        assert np.array_equal(got, np.argsort(x, kind="stable"))


@pytest.mark.parametrize("n", [4097, 250_007])
def test_two_keys_with_nulls(bolt, engine, n):
    """Row ids as payload and NULL rows split off, through both schedules (the first key has few digits)."""
    rng = np.random.default_rng(n)
    a = rng.integers(0, 50, n).astype(np.int32)
    b = _keys("full", n)
    valid = rng.random(n) > 0.1
    cols = [bolt.col(a, "i32", bitmap(valid)).to("cuda"), bolt.col(b).to("cuda")]
    got = engine.sort_indices(cols, [True, False], [False, False]).cpu().numpy().view(np.uint32)
    assert np.array_equal(got, np.lexsort((b, np.where(valid, -a, 0), ~valid)))


def test_many_segments(bolt, engine):
    """Segments of one batched GROUP BY finalize, each with its own schedule: keys in order, no group lost."""
    rng = np.random.default_rng(5)
    pqs, want = [], []
    for i, (n, groups) in enumerate([(60_000, 50_000), (300_000, 20_000), (300_000, 7_000), (9_000, 9_000)]):
        k = rng.integers(-(1 << 62), 1 << 62, groups)[rng.integers(0, groups, n)] >> (8 * i)
        pqs.append(engine.prepare_groupby({"k": bolt.col(k).to("cuda")}, ["k"], [("count_star", None)],
                                          groups_hint=groups))
        want.append(np.unique(k, return_counts=True))
    for r, (u, c) in zip(engine.execute_batch(pqs), want):
        assert np.array_equal(r.keys[0].numpy(), u) and np.array_equal(r.aggs[0].numpy(), c)
