"""The pooled traversal on boxes where its padding, batches and units can go wrong: sides below the halo
(several periodic copies), one cell wide, odd sides, ray counts around a batch of 32, several seeds, and
a long thin box that has no padded occupancy.  Counts and visited cells equal the oracle's."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import porerad_oracle as oracle

pytestmark = pytest.mark.gpu


def _box(shape, phi, seed):
    return (np.random.default_rng(seed).random(shape) < phi).astype(np.uint8)


def _check(ph, rays, seeds):
    from porerad_b200 import view_factors as vf

    want = oracle.build_surface_patches(ph, 0.01)
    p = vf.build_surface_patches(ph, 0.01)
    assert p.n_patches == want.n_patches
    stats = {}
    tables = [oracle.first_hit_counts(want, rays, s, stats=stats) for s in seeds]
    o, r, c = oracle.pool_counts(tables, want.n_patches)
    t = vf.first_hit_counts_pooled(p, rays, seeds)
    go, gr, gc = t.to_numpy()
    assert np.array_equal(go, o) and np.array_equal(gr, r) and np.array_equal(gc, c)
    assert t.dda_steps == stats["steps"] and t.rays_traced == stats["rays"]


@pytest.mark.parametrize("rays", [1, 31, 32, 33, 100])
@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 3, 2), (30, 1, 1), (9, 16, 15), (12, 17, 33), (33, 40, 7), (24, 32, 48)])
def test_counts_of_odd_boxes(shape, rays):
    ph = _box(shape, 0.15 if np.prod(shape) > 1 else 0.0, 3)
    if ph.size > 1:
        ph[:, 0, 0] = 0  # a straight pore through every box
    _check(ph, rays, [11])


@pytest.mark.parametrize("seeds", [[1, 2], [5, 6, 7]])
def test_counts_of_several_seeds(seeds):
    _check(_box((14, 13, 11), 0.1, 4), 37, seeds)


def test_counts_without_padded_occupancy():
    # 250000 x 2 x 2 cells: the padded copy would be 290 times as many; plugs every 40 cells
    ph = np.zeros((250_000, 2, 2), np.uint8)
    ph[20::40, :, :] = 1
    _check(ph, 2, [9])


def test_batches_of_boxes_with_and_without_padded_occupancy():
    """One long thin box among others: every table is the box's own, and the others are walked by the
    traversal variant that was asked for."""

    from porerad_b200 import _lib, view_factors as vf

    thin = np.zeros((250_000, 2, 2), np.uint8)
    thin[20::40, :, :] = 1
    boxes = [thin, _box((14, 13, 11), 0.1, 4), thin[:200_000], _box((9, 16, 15), 0.15, 5), _box((24, 32, 48), 0.1, 6)]
    patches = [vf.build_surface_patches(b, 0.01) for b in boxes]
    seeds = [[3, 4], [5, 6], [7, 8], [9, 10], [11, 12]]
    try:
        _lib.check(_lib.load().pr_trace_set_variant(2))
        batch = vf.first_hit_counts_batch(patches, 5, seeds)
        assert _lib.trace_variant()[0] == 2
    finally:
        _lib.load().pr_trace_set_variant(-1)
    for p, s, t in zip(patches, seeds, batch):
        one = vf.first_hit_counts_pooled(p, 5, s)
        assert t.dda_steps == one.dda_steps and t.rays_traced == one.rays_traced
        for a, b in zip(t.to_numpy(), one.to_numpy()):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("shape,plugs,rays,seeds", [
    ((400_000, 1, 1), 0, 33, [1]),  # two wall patches and nothing between them
    ((400_000, 1, 1), 7000, 31, [2, 3]), ((300_000, 3, 1), 900, 1, [4]), ((250_000, 2, 2), 60, 1, [5, 6]),
    ((110_000, 40, 8), 2000, 1, [7]),
])
def test_counts_of_boxes_without_padded_occupancy(shape, plugs, rays, seeds):
    """Their own walk: remainders of a batch, several seeds, one periodic cell, walls met by most rays."""

    ph = np.zeros(shape, np.uint8)
    if plugs:
        ph[20::plugs] = 1
        if shape[1] > 1:
            ph[21::plugs, 0, 0] = 1
            ph[23::plugs, 1 % shape[1], 0] = 1
    assert np.prod([shape[0] + 16, shape[1] + 32, shape[2] + 32]) > max(2**28, 4 * ph.size)
    _check(ph, rays, seeds)
