"""Pooling of edge lists: sorted lists (row merges), any other order, repeats, empty lists and counts that
only fit after pooling give the table of the oracle; what was refused stays refused."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import porerad_oracle as oracle

pytestmark = pytest.mark.gpu


def _list(n, m, rng, sort=True):
    key = np.unique(rng.integers(0, n * n, m))
    o, r = (key // n).astype(np.int32), (key % n).astype(np.int32)
    c = rng.integers(0, 9, key.size)
    if not sort:
        p = rng.permutation(key.size)
        o, r, c = o[p], r[p], c[p]
    return o, r, c.astype(np.int64)


def _check(tables, n):
    from porerad_b200 import view_factors as vf

    got, want = vf.pool_counts(tables, n), oracle.pool_counts(tables, n)
    for g, w in zip(got, want):
        assert g.dtype == w.dtype and np.array_equal(g, w)


@pytest.mark.parametrize("kinds", ["s", "u", "ss", "su", "us", "sss", "ses", "essu", "d", "sd"])
@pytest.mark.parametrize("n,m", [(1, 1), (7, 20), (300, 5000), (5000, 200000)])
def test_lists_of_every_form(n, m, kinds):
    rng = np.random.default_rng(len(kinds) + n)
    tables = []
    for k in kinds:
        if k == "e":
            tables.append(tuple(np.empty(0, t) for t in (np.int32, np.int32, np.int64)))
            continue
        t = _list(n, m, rng, sort=k != "u")
        if k == "d":  # every pair twice, still ascending
            t = tuple(np.repeat(a, 2) for a in t)
        tables.append(t)
    _check(tables, n)


def test_counts_that_cancel_and_counts_past_int32():
    from porerad_b200 import view_factors as vf

    a = (np.array([0, 1], np.int32), np.array([1, 0], np.int32), np.array([5, 2**31 + 4], np.int64))
    b = (np.array([0, 1], np.int32), np.array([1, 0], np.int32), np.array([-2, -(2**31)], np.int64))
    _check([a, b], 2)
    top = (np.array([0], np.int32), np.array([1], np.int32), np.array([2**31 - 1], np.int64))
    _check([top], 2)
    for tables in ([top, top], [a], [b]):
        with pytest.raises(ValueError, match="pooled counts"):
            vf.pool_counts(tables, 2)


@pytest.mark.parametrize("where", [0, 1])
@pytest.mark.parametrize("value", [-1, 4])
def test_ids_outside_are_refused(where, value):
    from porerad_b200 import view_factors as vf

    t = [np.array([0, 1, 2, 3], np.int32), np.array([1, 1, 1, 1], np.int32), np.ones(4, np.int64)]
    t[where][0 if value < 0 else 3] = value
    with pytest.raises(IndexError):
        vf.pool_counts([tuple(t)], 4)


@pytest.mark.parametrize("a,b", [(0, 1280), (640, 640), (640, 641), (1281, 0), (1280, 1), (3, 2500), (2500, 3), (33, 31)])
def test_rows_around_the_staged_length(a, b):
    """Row pairs that are merged in shared memory and those that are not, with columns in common."""

    n, rng = 3000, np.random.default_rng(a + b)
    tables = []
    for k in (a, b):
        rows = [np.sort(rng.choice(n, k, replace=False)) for _ in range(5)]
        o = np.repeat(np.arange(5) * 7, k).astype(np.int32)
        r = np.concatenate(rows).astype(np.int32)
        tables.append((o, r, rng.integers(1, 50, o.size).astype(np.int64)))
    _check(tables, n)


@pytest.mark.parametrize("lists,m", [(3, 530_000), (4, 800_000), (5, 1_100_000), (7, 1_800_000)])
def test_many_lists_by_merges(lists, m):
    """Lists long enough that three and more of them are merged, the odd one of a level passed on."""

    rng = np.random.default_rng(lists)
    tables = [_list(3000, m, rng) for _ in range(lists)]
    assert sum(t[0].size for t in tables) >= 250_000 * lists * (lists - 1)
    _check(tables, 3000)


@pytest.mark.parametrize("lists", [8, 17, 64])
def test_many_short_lists_do_not_cost_a_merge_each(lists):
    from porerad_b200 import _lib, view_factors as vf

    rng = np.random.default_rng(lists)
    tables = [_list(200, 300, rng) for _ in range(lists)]
    _check(tables, 200)  # loads and warms up
    before = _lib.load().pr_kernel_launches()
    _check(tables, 200)
    # one sort of all lists
    assert _lib.load().pr_kernel_launches() - before <= 10
    o, r, c = tables[lists // 2]
    for bad in (np.where(np.arange(o.size) == 5, 200, o), np.where(np.arange(o.size) == 5, -1, o)):
        with pytest.raises(IndexError, match="patch ids"):
            vf.pool_counts([*tables, (bad.astype(np.int32), r, c)], 200)
    with pytest.raises(IndexError, match="patch ids"):
        vf.pool_counts(tables, 0)
