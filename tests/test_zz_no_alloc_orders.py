"""soil_bin_sort_noalloc on inputs in nearly sorted order and in crowded cells,
where a warp counts its cells together: against a stable argsort, on both sides
of the number of alike neighbours that decides, with ragged ends, and with more
atoms in a cell than the bits beside its number count."""
import numpy as np
import pytest

from test_zz_no_alloc_forms import _check

pytestmark = pytest.mark.gpu


# mean atoms per cell around the 16 of 31 neighbours that share a cell
@pytest.mark.parametrize("per_cell", [0.7, 1.5, 2.0, 2.5, 4, 30, 300])
@pytest.mark.parametrize("n", [33, 1021, 40007])
def test_nearly_sorted_orders(ctx, per_cell, n):
    rng = np.random.default_rng(n)
    m = max(1, round((n / per_cell) ** (1 / 3)))
    pos = rng.random((n, 3)) * m
    k = np.floor(pos).astype(np.int64)
    order = np.argsort((k[:, 0] * m + k[:, 1]) * m + k[:, 2], kind="stable")
    _check(ctx, pos[order], (m, m, m))
    _check(ctx, pos[order[::-1]], (m, m, m))
    _check(ctx, np.clip(pos[order] + rng.normal(0.0, 0.05, (n, 3)), 0.0, m - 1e-9), (m, m, m))
    swapped = order.copy()  # every other atom from elsewhere
    swapped[1::2] = rng.permutation(swapped[1::2])
    _check(ctx, pos[swapped], (m, m, m))


def test_sorted_cells_of_more_atoms_than_their_places_count(ctx):
    rng = np.random.default_rng(5)
    parts = [np.array([c, 1.0, 2.0]) + rng.random((k, 3))
             for c, k in ((0.0, 2400), (1.0, 2047), (2.0, 2048), (3.0, 5), (4.0, 3001))]
    pos = np.concatenate(parts)
    _check(ctx, pos, (5, 3, 3))
    _check(ctx, pos[::-1], (5, 3, 3))
    mixed = pos.copy()
    mixed[::3] = pos[::3][rng.permutation(len(pos[::3]))]
    _check(ctx, mixed, (5, 3, 3))
