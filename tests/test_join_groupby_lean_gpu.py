"""The dense join GROUP BY kernel against numpy, exactly: key and value types, payloads around -1, group counts
from one to past the shared and the first global table, row counts off every tile and step."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 1,024 rows: one CTA's step; 148 x 2 x 1,024 rows: the whole grid's.
@pytest.mark.parametrize("n,groups", [(1, 1), (1023, 3), (1025, 100), (303_105, 1000), (2_000_003, 1500),
                                      (1_000_001, 20_000)])
@pytest.mark.parametrize("kdt,vdt", [("i64", "dec128"), ("i32", "dec128"), ("i64", "i64"), ("i32", "i32")])
def test_against_numpy(bolt, engine, kdt, vdt, n, groups):
    rng = np.random.default_rng(n + groups)
    np_k = np.int64 if kdt == "i64" else np.int32
    nb = 40_000
    bk = rng.permutation(np.arange(-1, nb - 1)).astype(np_k) * np_k(1 if kdt == "i32" else 1 << 40)
    bg = rng.integers(-2, groups - 2, nb).astype(np.int32)  # -1: the payload whose complement is 0
    pick = rng.integers(0, nb + 4000, n)  # the last 4,000 match nothing
    pk = np.where(pick < nb, bk[np.minimum(pick, nb - 1)], np_k(nb + 7)).astype(np_k)
    v = rng.integers(-2**31, 2**31, n) if vdt == "i32" else rng.integers(-2**40, 2**40, n)
    if vdt == "dec128":
        col = bolt.col(np.stack([v, v >> 63], axis=1), "dec128")
    else:
        col = bolt.col(v.astype(np.int32 if vdt == "i32" else np.int64), vdt)
    g, s, c = engine.join_groupby(bolt.col(bk, kdt).to("cuda"), bolt.col(bg, "i32").to("cuda"),
                                  bolt.col(pk, kdt).to("cuda"), col.to("cuda"))
    hit = pick < nb
    pg = bg[pick[hit]]
    ug, inv = np.unique(pg, return_inverse=True)
    sums = np.zeros(len(ug), np.int64)
    np.add.at(sums, inv, v[hit])
    assert np.array_equal(g.numpy(), ug)
    assert np.array_equal(c.numpy(), np.bincount(inv, minlength=len(ug)))
    got = s.numpy()
    if vdt == "dec128":
        assert np.array_equal(got[:, 1], got[:, 0] >> 63)
        got = got[:, 0]
    assert np.array_equal(got, sums)
