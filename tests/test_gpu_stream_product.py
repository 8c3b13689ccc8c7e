"""Products of operators stored as word streams, on count tables made to reach the edges of the layout: one
row, rows below and above a quad, a row long enough to pass through several warps of a stage, rows
without entries in most column blocks, patch counts around a column block, the ray counts from which a
pair's count may take several words, and the sizes at which the plain storage takes over.

Every row sum has at most m = 2 (longest row) terms of one sign, so any order of summation is within
m 2^-53 of the exact sum, relative to it; two such sums and the scalings are within (2 m + 8) 2^-53.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _table(n, kind, rays, rng):
    """(origin, receiver, count) with every row summing to `rays`."""

    o, r, c = [], [], []
    for i in range(n):
        if kind == "self":
            cols = np.array([i])
        elif kind == "band":
            cols = np.unique((i + np.arange(-2, 3)) % n)
        elif kind == "long" and i % 1000 == 3:
            cols = np.arange(n)
        elif kind == "far":
            cols = np.unique(np.array([i, (i * 7919) % n, n - 1 - i]))
        else:
            cols = np.unique(rng.integers(0, n, int(rng.integers(1, 40))))
        cols = cols[:rays]
        cnt = np.ones(cols.size, np.int64)
        cnt[int(rng.integers(0, cols.size))] += rays - cols.size
        o.append(np.full(cols.size, i))
        r.append(cols)
        c.append(cnt)
    return (np.concatenate(o).astype(np.int32), np.concatenate(r).astype(np.int32), np.concatenate(c))


def _symmetric(n, o, r, c, rays, area):
    from scipy.sparse import coo_matrix

    F = coo_matrix((c / rays, (o, r)), shape=(n, n)).tocsr()
    S = 0.5 * area * (F + F.T)
    return S.tocsr(), int(np.max(np.diff(S.indptr)))


@pytest.mark.parametrize("n,kind,rays", [
    (1, "self", 3), (2, "band", 4), (31, "random", 50), (148, "self", 65535), (149, "band", 7), (1024, "random", 64),
    (4100, "long", 4200), (16384, "far", 9), (16385, "band", 100), (30011, "random", 333), (70000, "far", 65536),
])
def test_products_and_balancing(n, kind, rays):
    from porerad_b200 import exchange

    rng = np.random.default_rng(n + rays)
    o, r, c = _table(n, kind, rays, rng)
    area = np.full(n, 0.75)
    if rays == 65536:  # three nearly disjoint permutations: no positive diagonal balances them, in any storage
        with pytest.raises(RuntimeError, match="balancing"):
            exchange.ExchangeOperator(o, r, c, np.full(n, rays, np.int64), area)
        return
    op = exchange.ExchangeOperator(o, r, c, np.full(n, rays, np.int64), area)
    S, longest = _symmetric(n, o, r, c, rays, 0.75)
    bound = (4 * longest + 8) * 2.0**-53
    x = rng.random(n) + 0.5
    want = S @ x + 1e-15 * area * x
    got = op.symmetric_matvec(x)
    assert np.max(np.abs(got - want) / want) <= bound
    assert np.array_equal(got, op.symmetric_matvec(x))
    # d (S d) = A to the balancing tolerance, and F_p x from the same products
    assert np.max(np.abs(op.scale * (S @ op.scale + 1e-15 * area * op.scale) / area - 1.0)) <= 1e-10 + bound
    d = op.scale
    want = d / area * (S @ (d * x) + 1e-15 * area * d * x)
    assert np.max(np.abs(op.matvec(x) - want) / want) <= bound + 2.0**-50


@pytest.mark.parametrize("n", [300, 20000])
def test_batched_operators_equal_single_ones(n):
    from porerad_b200 import exchange, view_factors as vf

    rng = np.random.default_rng(n)
    args = [(*_table(k, "random", 80, rng), k) for k in (n, n // 3, n + 17)]
    tables = [vf.pool_to_device(o, r, c, k) for o, r, c, k in args]
    rays = [np.full(k, 80, np.int64) for *_, k in args]
    areas = [np.full(k, 0.5) for *_, k in args]
    batch = exchange.ExchangeOperator.from_tables(tables, rays, areas)
    for op, t, q, a in zip(batch, tables, rays, areas):
        one = exchange.ExchangeOperator(t, None, None, q, a)
        assert np.array_equal(op.scale, one.scale) and op.balance_iterations == one.balance_iterations


@pytest.mark.parametrize("n", [50, 20001])
def test_binary32_sweeps_reach_the_binary64_series(n):
    """The mixed solve's binary32 products on the same stream: net powers of the two precisions."""

    from porerad_b200 import coupled, exchange, view_factors as vf

    rng = np.random.default_rng(1)
    ph = (rng.random((8, 8, 8) if n < 100 else (40, 36, 33)) < 0.12).astype(np.uint8)
    p = vf.build_surface_patches(ph, 0.01)
    t = vf.first_hit_counts_pooled(p, 50, [3])
    op = exchange.ExchangeOperator(t, None, None, np.full(p.n_patches, 50, np.int64), np.asarray(p.patch_area_m2))
    a = coupled.prescribed_field_channels(op, p, 700.0, 50.0, 0.4)
    b = coupled.prescribed_field_channels(op, p, 700.0, 50.0, 0.4, precision="mixed")
    scale = max(abs(a.q_h), abs(a.q_c), abs(a.q_i))
    assert max(abs(a.q_h - b.q_h), abs(a.q_c - b.q_c), abs(a.q_i - b.q_i)) <= 1e-8 * scale


@pytest.mark.parametrize("n", [40, 20011])
def test_infinities_and_nans_stay_in_their_rows(n):
    """A value of x that is not finite reaches the rows that have its column, and no others."""

    from porerad_b200 import exchange

    o, r, c = _table(n, "band", 20, np.random.default_rng(4))
    op = exchange.ExchangeOperator(o, r, c, np.full(n, 20, np.int64), np.full(n, 0.5))
    S, _ = _symmetric(n, o, r, c, 20, 0.5)
    for value, columns in ((np.inf, (0, 7)), (np.nan, (0, n - 1))):
        x = np.ones(n)
        x[list(columns)] = value
        touched = np.asarray((S[:, list(columns)] != 0).sum(axis=1)).ravel() > 0
        assert np.array_equal(~np.isfinite(op.symmetric_matvec(x)), touched)


@pytest.mark.parametrize("n,kind", [
    (12224, "random"), (12225, "random"), (12225, "self"), (24449, "long"), (61000, "band"),
    (110016, "random"), (110017, "random"),
])
def test_column_groups(n, kind):
    """Patch counts around a column group and around the most sums that products in groups leave, tables
    with most rows of a group empty, and the sums taken over the groups of every row."""

    from porerad_b200 import exchange

    rays = n + 1 if kind == "long" else 60
    rng = np.random.default_rng(n)
    o, r, c = _table(n, kind, rays, rng)
    op = exchange.ExchangeOperator(o, r, c, np.full(n, rays, np.int64), np.full(n, 0.75))
    S, longest = _symmetric(n, o, r, c, rays, 0.75)
    bound = (4 * longest + 8) * 2.0**-53
    x = rng.random(n) + 0.5
    want = S @ x + 1e-15 * 0.75 * x
    got = op.symmetric_matvec(x)
    assert np.max(np.abs(got - want) / want) <= bound
    assert np.array_equal(got, op.symmetric_matvec(x))
    assert np.max(np.abs(op.scale * (S @ op.scale + 1e-15 * 0.75 * op.scale) / 0.75 - 1.0)) <= 1e-10 + bound
    x[5] = np.nan
    touched = np.asarray((S[:, [5]] != 0).sum(axis=1)).ravel() > 0
    touched[5] = True  # the support diagonal 1e-15 A
    assert np.array_equal(np.isnan(op.symmetric_matvec(x)), touched)


@pytest.mark.parametrize("n", [330_000, 400_000, 1_300_000])
def test_many_patches_with_short_rows(n):
    """Patch counts below and above those at which short rows leave the stream, whose padding grows with
    the square of the patches: an operator takes at most 1000 bytes a patch here (columns, counts and their
    transpose at most 16 bytes an entry, five entries a patch, 41 quads, and 100 bytes a patch for the
    vectors and offsets, in blocks rounded up by an eighth)."""

    from scipy.sparse import coo_matrix

    from porerad_b200 import _lib, exchange, view_factors as vf

    rays = 9
    i = np.arange(n, dtype=np.int64)
    c = np.sort((i[:, None] + np.arange(-2, 3)) % n, axis=1)
    o = np.repeat(i, 5).astype(np.int32)
    cnt = np.where(c == i[:, None], rays - 4, 1).ravel().astype(np.int64)
    c = c.ravel().astype(np.int32)
    table = vf.pool_to_device(o, c, cnt, n)
    area = np.full(n, 0.75)
    before = _lib.memory_stats()["live_bytes"]
    op = exchange.ExchangeOperator(table, None, None, np.full(n, rays, np.int64), area)
    assert _lib.memory_stats()["live_bytes"] - before <= 1000 * n
    F = coo_matrix((cnt / rays, (o, c)), shape=(n, n)).tocsr()
    S = (0.5 * 0.75 * (F + F.T)).tocsr()
    bound = (4 * 5 + 8) * 2.0**-53
    x = np.random.default_rng(n).random(n) + 0.5
    want = S @ x + 1e-15 * 0.75 * x
    assert np.max(np.abs(op.symmetric_matvec(x) - want) / want) <= bound
    d = op.scale
    assert np.max(np.abs(d * (S @ d + 1e-15 * area * d) / area - 1.0)) <= 1e-10 + bound
    small = _table(300, "random", 80, np.random.default_rng(1))
    tables = [table, vf.pool_to_device(*small, 300)]
    batch = exchange.ExchangeOperator.from_tables(tables, [np.full(n, rays, np.int64), np.full(300, 80, np.int64)],
                                                  [area, np.full(300, 0.5)])
    assert np.array_equal(batch[0].scale, d) and np.array_equal(batch[0].symmetric_matvec(x), op.symmetric_matvec(x))


def _wide_table(n, rays, rng):
    """Rows of 20 to 40 columns, 0.3 of the rays to one of them: every table balances."""

    o, r, c = [], [], []
    for i in range(n):
        cols = np.unique(rng.integers(0, n, int(rng.integers(20, 41))))
        w = np.full(cols.size, 0.7 / cols.size)
        w[int(rng.integers(0, cols.size))] += 0.3
        o.append(np.full(cols.size, i))
        r.append(cols)
        c.append(1 + rng.multinomial(rays - cols.size, w))
    return (np.concatenate(o).astype(np.int32), np.concatenate(r).astype(np.int32), np.concatenate(c).astype(np.int64))


@pytest.mark.parametrize("n", [2000, 20011])
@pytest.mark.parametrize("rays", [65535, 65536, 600_000, 50_000_000, 1_000_000_000])
def test_ray_counts_past_a_word(n, rays):
    """Ray counts around those whose pair counts fit a word, those where some counts are split over several
    words, and those where most would be: products, balancing and the infinities' rows."""

    from porerad_b200 import exchange

    rng = np.random.default_rng(n + rays)
    o, r, c = _wide_table(n, rays, rng)
    op = exchange.ExchangeOperator(o, r, c, np.full(n, rays, np.int64), np.full(n, 0.75))
    S, longest = _symmetric(n, o, r, c, rays, 0.75)
    assert op.nnz == c.size and op.nnz_symmetric == S.nnz
    # a row's pieces: its entries and one for every 2^17 - 1 of its pairs
    pairs = np.bincount(o, c, n) + np.bincount(r, c, n)
    terms = longest + (int(pairs.max()) // (2**17 - 1) if rays < 10**6 else 0)
    bound = (4 * terms + 8) * 2.0**-53
    x = rng.random(n) + 0.5
    want = S @ x + 1e-15 * 0.75 * x
    got = op.symmetric_matvec(x)
    assert np.max(np.abs(got - want) / want) <= bound
    assert np.array_equal(got, op.symmetric_matvec(x))
    d = op.scale
    assert np.max(np.abs(d * (S @ d + 1e-15 * 0.75 * d) / 0.75 - 1.0)) <= 1e-10 + bound
    x[5] = np.inf
    touched = np.asarray((S[:, [5]] != 0).sum(axis=1)).ravel() > 0
    touched[5] = True  # the support diagonal 1e-15 A
    assert np.array_equal(np.isinf(op.symmetric_matvec(x)), touched)


def test_batches_past_a_word_share_their_launches():
    """Operators of 65536 rays are balanced in the launches of one batch, as those of 65535 are."""

    from porerad_b200 import _lib, exchange, view_factors as vf

    launches = {}
    for rays in (65535, 65536):
        rng = np.random.default_rng(3)
        tables = [vf.pool_to_device(*_wide_table(n, rays, rng), n) for n in (500, 501, 502, 503, 504, 505)]
        sizes = [t.n_patches for t in tables]
        before = _lib.load().pr_kernel_launches()
        ops = exchange.ExchangeOperator.from_tables(tables, [np.full(n, rays, np.int64) for n in sizes],
                                                    [np.full(n, 0.5) for n in sizes])
        launches[rays] = _lib.load().pr_kernel_launches() - before
        for op, t, n in zip(ops, tables, sizes):
            one = exchange.ExchangeOperator(t, None, None, np.full(n, rays, np.int64), np.full(n, 0.5))
            assert np.array_equal(op.scale, one.scale)
    # two more launches an operator look for counts to split; a table's iterations may differ by a few
    assert launches[65536] <= launches[65535] + 6 * 2 + 24


def test_many_rows_of_one_entry_beside_long_ones():
    """Rows so uneven that equal shares of the entries would give one CTA most of the rows: 6 500 patches
    that see themselves alone beside 5 600 that see a quarter of each other."""

    from porerad_b200 import exchange

    n, alone, rays = 12_100, 6_500, 1_500
    rng = np.random.default_rng(8)
    o, r, c = [np.arange(alone)], [np.arange(alone)], [np.full(alone, rays)]
    for i in range(alone, n):
        cols = alone + np.sort(rng.choice(n - alone, 1_400, replace=False))
        cnt = np.ones(cols.size, np.int64)
        cnt[:100] += 1
        o.append(np.full(cols.size, i))
        r.append(cols)
        c.append(cnt)
    o, r, c = np.concatenate(o).astype(np.int32), np.concatenate(r).astype(np.int32), np.concatenate(c).astype(np.int64)
    op = exchange.ExchangeOperator(o, r, c, np.full(n, rays, np.int64), np.full(n, 0.75))
    S, longest = _symmetric(n, o, r, c, rays, 0.75)
    x = rng.random(n) + 0.5
    want = S @ x + 1e-15 * 0.75 * x
    assert np.max(np.abs(op.symmetric_matvec(x) - want) / want) <= (4 * longest + 8) * 2.0**-53
