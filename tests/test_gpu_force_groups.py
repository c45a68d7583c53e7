"""The consumer queued before the pair total is known, and its form with 8
lanes per root: forces (ghosts' included) equal the CPU oracle's at the sizes
around its line, with roots of 0 to 26 images, and when the early launch finds
its arrays too small or the ghosts outgrow theirs."""
import numpy as np
import pytest

import oracle
from helpers import assert_same_lists, assert_same_state
from soil_b200 import system, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [20, 31, 200, 1000, 18945, 37888, 37889, 60000])
@pytest.mark.parametrize("newton", [1, 0])
@pytest.mark.parametrize("rate", [0.0, 0.3])
def test_rebuild_step_forces_match_oracle(ctx, n, newton, rate):
    w = W.poly("groups", 200 + n % 3, n, 0.5, 1e-4, 0, harmonic_k=1e3, newton=newton,
               shear_rate=rate)
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    for k in (1, 2):
        g.step(k)
        o.step(k)
        assert_same_state(g, o, f"n={n} step {k}")
        assert_same_lists(g, o)
    g.close()


def test_lists_and_ghosts_that_outgrow_their_arrays(ctx):
    """A sheared cloud that contracts: every step rebuilds, pairs grow past
    the arrays of the early launches."""
    w = W.poly("grow", 210, 4000, 0.12, 1e-3, 0, harmonic_k=1.0, shear_rate=0.05)
    w.vel[:] = (0.5 * w.L - w.pos) * 6.0
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    seen = 0
    for _ in range(12):
        g.step(10)
        o.step(10)
        assert_same_state(g, o)
        seen = max(seen, g.counts().npairs)
    assert seen > 2 * 4000
    assert_same_lists(g, o)
    g.close()


# The border pass with and without a scan of its own (up to 1,024 tiles of 32
# locals without), around its tiles' and CTAs' edges.
@pytest.mark.parametrize("n", [3, 8, 33, 255, 257, 8192, 8193, 32768, 32769])
def test_border_pass_of_few_and_many_tiles(ctx, n):
    w = W.poly("border-tiles", 210, n, 0.3, 1e-4, 0, harmonic_k=1e2)
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    g.step(2)
    o.step(2)
    assert_same_state(g, o, f"n={n}")
    assert_same_lists(g, o)
    for a, b in zip(g.swaps(), o.swaps()):
        assert a["recv_start"] == b["recv_start"] and a["recv_count"] == b["recv_count"]
        np.testing.assert_array_equal(a["send"], b["send"])
    g.close()
