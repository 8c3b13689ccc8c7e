"""The coupled solve on recycled device memory that holds NaNs."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operator(ph, rays):
    from porerad_b200 import exchange, view_factors as vf

    p = vf.build_surface_patches(ph, 0.01)
    t = vf.first_hit_counts_pooled(p, rays, [5])
    return p, exchange.ExchangeOperator(t, None, None, np.full(p.n_patches, rays, np.int64), np.asarray(p.patch_area_m2))


def test_coupled_solve_does_not_read_recycled_memory():
    """The Krylov basis (31 vectors of the cells) is one allocation; a cell field of NaNs on a box of 31 times
    the cells leaves a released block of that size full of them for it."""

    from porerad_b200 import conduction, coupled

    rng = np.random.default_rng(2)
    ph = (rng.random((12, 12, 12)) < 0.15).astype(np.uint8)
    p, op = _operator(ph, 100)
    system = conduction.assemble_conduction(np.where(ph == 1, 0.2, 0.026), 0.01)
    T0 = conduction.solve_conduction(system, 710.0, 690.0)
    first = coupled.solve_coupled(system, op, p, 710.0, 690.0, 0.6, T0)
    big = (rng.random((31 * 12, 12, 12)) < 0.15).astype(np.uint8)
    pb, opb = _operator(big, 50)
    with pytest.raises(RuntimeError, match="series"):
        coupled.cell_field_channels(opb, pb, np.full(big.shape, np.nan), 710.0, 690.0, 0.6)
    again = coupled.solve_coupled(system, op, p, 710.0, 690.0, 0.6, T0)
    assert first.converged and again.converged
    assert np.array_equal(first.temperature_K, again.temperature_K)
