"""soil_bin_sort_noalloc against a stable argsort: atom counts and grids around
the edges of its passes, atoms in random order and in cell order, and cells
that hold more atoms than the bits beside a cell number count."""
import ctypes as C

import numpy as np
import pytest
import torch

from soil_b200 import abi

pytestmark = pytest.mark.gpu


def _sort(ctx, pos, count):
    f3, i3 = C.c_double * 3, C.c_int32 * 3
    dev = [torch.tensor(pos[:, d].copy(), device="cuda") for d in range(3)]
    n = len(pos)
    out = torch.full((2, max(n, 1)), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    st = ctx.lib.soil_bin_sort_noalloc(
        ctx.h, *[C.c_void_p(t.data_ptr()) for t in dev], n, f3(0, 0, 0), f3(1, 1, 1), i3(*count),
        f3(0, 0, 0), f3(*[float(c) for c in count]), f3(0, 0, 0), 0, C.c_void_p(out[0].data_ptr()),
        C.c_void_p(out[1].data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == abi.SOIL_OK, ctx.error()
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _check(ctx, pos, count):
    cell, perm = _sort(ctx, pos, count)
    k = np.clip(np.floor(pos).astype(np.int64), 0, np.array(count) - 1)
    want = (k[:, 0] * count[1] + k[:, 1]) * count[2] + k[:, 2]
    np.testing.assert_array_equal(cell[:len(pos)], want)
    np.testing.assert_array_equal(perm[:len(pos)], np.argsort(want, kind="stable"))


@pytest.mark.parametrize("n", [1, 31, 257, 70001])
@pytest.mark.parametrize("count", [(1, 1, 1), (3, 5, 7), (64, 64, 32), (50, 52, 53), (128, 128, 128)])
def test_sizes_and_grids(ctx, n, count):
    if n > 300 * count[0] * count[1] * count[2]:
        n = 300 * count[0] * count[1] * count[2]
    rng = np.random.default_rng(n + count[2])
    pos = rng.random((n, 3)) * np.array(count)
    _check(ctx, pos, count)
    _check(ctx, pos[np.argsort(pos[:, 0], kind="stable")], count)


def test_more_atoms_in_a_cell_than_its_places_count(ctx):
    rng = np.random.default_rng(3)
    crowd = np.array([2.0, 3.0, 4.0]) + rng.random((2400, 3))
    edge = np.array([0.0, 0.0, 0.0]) + rng.random((2047, 3))
    more = np.array([5.0, 5.0, 5.0]) + rng.random((2048, 3))
    pos = np.concatenate([crowd, edge, more, rng.random((4000, 3)) * 8.0])
    _check(ctx, pos[rng.permutation(len(pos))], (8, 8, 8))
