"""Aggregate layouts with a row loop of their own (SUM alone, several SUM / AVG, COUNT(*) beside a nullable SUM),
through every kernel that serves them, against the oracle; with and without WHERE, at sizes around the streaming
kernel's start and off every tile."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from helpers import bitmap
from test_groupby_gpu import run_both

pytestmark = pytest.mark.gpu

LAYOUTS = {"sum_i64": [("sum", "v")], "sum_f64": [("sum", "x")], "sum_i32": [("sum", "w")],
           "avg2": [("avg", "x"), ("avg", "y")], "avg3": [("avg", "x"), ("sum", "y"), ("avg", "z")],
           "sum2_i64": [("sum", "v"), ("sum", "u")],
           "count_sum_nullable_f64": [("sum", "xn"), ("count_star", None)],
           "count_avg_nullable_i64": [("count_star", None), ("avg", "vn")]}


def _columns(n, groups, seed):
    r = np.random.default_rng(seed)
    ok = bitmap(r.random(n) > 0.2)
    return {"k": (r.integers(-groups, groups, n).astype(np.int32), None, "i32", 0),
            "l": (r.integers(-groups, groups, n) * (1 << 33), None, "i64", 0),
            "m": (r.integers(0, 3, n).astype(np.int32), None, "i32", 0),
            "f": (r.integers(0, 100, n).astype(np.int32), None, "i32", 0),
            "v": (r.integers(-10**6, 10**6, n), None, "i64", 0), "u": (r.integers(-2**40, 2**40, n), None, "i64", 0),
            "w": (r.integers(-2**31, 2**31, n).astype(np.int32), None, "i32", 0),
            "x": (r.normal(0, 1e3, n), None, "f64", 0), "y": (r.normal(5, 1e-3, n), None, "f64", 0),
            "z": (r.normal(0, 1e8, n), None, "f64", 0), "xn": (r.normal(0, 10, n), ok, "f64", 0),
            "vn": (r.integers(-9, 9, n), ok, "i64", 0)}


# 262,144 rows: the streaming kernel's start; 31 x 64 rows: its tile; 64 rows: one warp's share.
@pytest.mark.parametrize("n,groups", [(1, 1), (20_011, 50), ((1 << 18) - 1, 3), ((1 << 18) + 1, 700),
                                      (31 * 64 * 148 + 65, 40_000)])
@pytest.mark.parametrize("layout", LAYOUTS)
def test_layouts(bolt, engine, oracle, layout, n, groups):
    cols = _columns(n, groups, n + groups)
    for keys in (["k"], ["l"], ["k", "m"]):
        run_both(bolt, engine, oracle, cols, keys, LAYOUTS[layout], hint=2 * groups)
        run_both(bolt, engine, oracle, cols, keys, LAYOUTS[layout], where=[("f", ">=", 40)], hint=2 * groups)


@pytest.mark.parametrize("kernel", ["regs", "staged", "part"])
@pytest.mark.parametrize("layout", LAYOUTS)
def test_layouts_on_every_kernel(bolt, engine, oracle, layout, kernel):
    flags = {"regs": bolt.FLAG_KERNEL_REGS, "staged": bolt.FLAG_KERNEL_STAGED, "part": bolt.FLAG_FORCE_PART}[kernel]
    run_both(bolt, engine, oracle, _columns(500_003, 20_000, 7), ["k", "m"], LAYOUTS[layout], where=[("f", "<", 70)],
             hint=100_000, flags=flags)


def test_layouts_share_a_batch(bolt, engine, oracle):
    """One batch of every layout: grouped by layout, each equal to its query alone."""
    cols = _columns(120_001, 300, 11)
    dev = {k: bolt.col(d, dt, v, s).to("cuda") for k, (d, v, dt, s) in cols.items()}
    pqs = [engine.prepare_groupby(dev, ["k"], a, groups_hint=700, rows=(100 * i, 120_001 - 1001 * i))
           for i, a in enumerate(LAYOUTS.values())]
    got = engine.execute_batch(pqs)
    for i, (a, r) in enumerate(zip(LAYOUTS.values(), got)):
        alone = engine.execute_batch([engine.prepare_groupby(dev, ["k"], a, groups_hint=700,
                                                             rows=(100 * i, 120_001 - 1001 * i))])[0]
        assert r.n_groups == alone.n_groups
        for x, y in zip(r.keys + r.aggs, alone.keys + alone.aggs):
            assert np.array_equal(x.numpy(), y.numpy(), equal_nan=x.dtype == "f64")


@pytest.mark.parametrize("n,count,own", [(3_000, 8, False), (900_000, 8, False), (1 << 20, 8, True), (400_000, 2, False),
                                         (900_000, 2, True), (3_000, 1, True)])
def test_batch_launches(bolt, engine, n, count, own):
    """A batch of several layouts costs one aggregation launch where they have few rows, and one a layout where the
    row loops compiled for them pay for it."""
    cols = _columns(n, 50, n)
    dev = {k: bolt.col(d, dt, v, s).to("cuda") for k, (d, v, dt, s) in cols.items()}

    def launches(layouts):
        engine.execute_batch([engine.prepare_groupby(dev, ["k"], a, groups_hint=101) for a in layouts])
        return engine.last_launches

    some = list(LAYOUTS.values())[:count]
    assert launches(some) - launches([some[0]] * count) == (count - 1 if own else 0)


@pytest.mark.parametrize("layout,tier", [("sum_i64", 1), ("avg3", 1), ("sum2_i64", 1), ("count_avg", 2)])
def test_partitioned_tier_on_request(bolt, engine, layout, tier):
    """The partitioned tier is asked for, but serves only the layouts it compiles; another one is planned for the
    global table straight away: as many graph nodes when captured as without the request."""
    from cuda.bindings import runtime as rt

    n = 500_003
    dev = {k: bolt.col(d, dt, v, s).to("cuda") for k, (d, v, dt, s) in _columns(n, 20_000, 3).items()}
    aggs = {**LAYOUTS, "count_avg": [("count_star", None), ("avg", "x")]}[layout]
    pq = engine.prepare_groupby(dev, ["k"], aggs, groups_hint=100_000)
    engine.execute_batch([pq])

    def nodes(flags):
        graph, stream = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            st = engine._lib.bolt_groupby(engine._ctx, C.byref(pq.desc), C.byref(pq.out), flags | bolt.FLAG_ASYNC,
                                          C.c_void_p(stream.cuda_stream))
        assert st == 0 and engine.last_groupby_tier == (tier if flags else 1)
        err, _, count = rt.cudaGraphGetNodes(rt.cudaGraph_t(graph.raw_cuda_graph()))
        assert err == rt.cudaError_t.cudaSuccess
        return count

    plain = [nodes(0), nodes(0)][1]  # (a kernel's first use can add one)
    asked = [nodes(bolt.FLAG_FORCE_PART), nodes(bolt.FLAG_FORCE_PART)][1]
    assert (asked == plain) == (tier == 1)
