"""Pass 1 of the pair build in each of its forms (8, 4 or 1 lanes per row, one
or two candidates at a time, forward and full stencils): rows and their order
equal the CPU oracle's, and the filter statistics those of the one-loop scan
(SOIL_PAIRS_PRE=0)."""
import os

import pytest

import oracle
from helpers import assert_same_lists, assert_same_state
from soil_b200 import abi, system, workloads as W

pytestmark = pytest.mark.gpu

# n on both sides of the lanes-per-row lines; phi on both sides of the
# two-at-a-time line, and packings whose rows are longer than their slots
CASES = [(33, 0.45), (12288, 0.45), (12289, 0.25), (36864, 0.3), (36865, 0.2), (36865, 0.5),
         (5000, 3.0), (40000, 3.0)]


def _stats(ctx, w, pre):
    old = os.environ.get("SOIL_PAIRS_PRE")
    os.environ["SOIL_PAIRS_PRE"] = pre
    try:
        g = system.from_workload(ctx, w)
        g.step(1)
        g.sync()
        c = g.counts()
        g.close()
        return c.npairs, c.filter_candidates, c.filter_rechecked
    finally:
        if old is None:
            del os.environ["SOIL_PAIRS_PRE"]
        else:
            os.environ["SOIL_PAIRS_PRE"] = old


@pytest.mark.parametrize("n,phi", CASES)
@pytest.mark.parametrize("newton", [1, 0])
@pytest.mark.parametrize("kind", ["poly", "mono", "poly-fp32", "mono-fp32"])
def test_rows_match_oracle(ctx, n, phi, newton, kind):
    make = W.poly if kind.startswith("poly") else W.mono
    kw = dict(filter=abi.SOIL_FILTER_FP32_RECHECK) if kind.endswith("fp32") else {}
    w = make("rows", 180, n, phi, 1e-5, 0, harmonic_k=1e2, newton=newton, **kw)
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    g.step(1)
    o.step(1)
    assert_same_state(g, o, f"{kind} n={n}")
    assert_same_lists(g, o)
    g.close()
    assert _stats(ctx, w, "1") == _stats(ctx, w, "0")


@pytest.mark.parametrize("n", [700, 2500, 9000, 60000, 110000])
@pytest.mark.parametrize("limit", [None, "8192"])
def test_scans_of_every_form(ctx, n, limit):
    """Count scans of one tile, of several tiles in one launch, of two
    launches, and pairs of scans on either side of the line."""
    old = os.environ.get("SOIL_SCAN1P_MAX")
    if limit:
        os.environ["SOIL_SCAN1P_MAX"] = limit
    try:
        w = W.poly("scans", 190, n, 0.4, 1e-4, 0, harmonic_k=1e3)
        g, o = system.from_workload(ctx, w), oracle.from_workload(w)
        g.step(2)
        o.step(2)
        assert_same_state(g, o, f"n={n}")
        assert_same_lists(g, o)
        g.close()
    finally:
        if limit:
            os.environ.pop("SOIL_SCAN1P_MAX") if old is None else os.environ.update(SOIL_SCAN1P_MAX=old)


# Pass 2 by 8 lanes per row up to 65,536 rows, and rows longer than their slots
# in it; the consumer of the step sorts the transposed lists.
@pytest.mark.parametrize("n,phi", [(3, 0.3), (7, 0.45), (33, 3.0), (3000, 6.0), (65536, 0.4),
                                   (65537, 0.4)])
@pytest.mark.parametrize("newton", [1, 0])
def test_rows_filled_by_lanes(ctx, n, phi, newton):
    w = W.poly("fill", 200, n, phi, 1e-5, 0, harmonic_k=1e2, newton=newton)
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    g.step(3)
    o.step(3)
    assert_same_state(g, o, f"n={n} phi={phi}")
    assert_same_lists(g, o)
    g.close()


# Stencils of every length: a box sheared until its full stencil has more runs
# than a row keeps in registers.
@pytest.mark.parametrize("n", [33, 3001, 40001])
@pytest.mark.parametrize("newton", [1, 0])
@pytest.mark.parametrize("kind", ["poly", "mono-fp32"])
def test_rows_of_strongly_tilted_boxes(ctx, n, newton, kind):
    make = W.poly if kind == "poly" else W.mono
    kw = dict(filter=abi.SOIL_FILTER_FP32_RECHECK) if kind.endswith("fp32") else {}
    w = make("tilted", 220, n, 0.4, 1e-4, 0, harmonic_k=1e2, shear_rate=150.0, newton=newton, **kw)
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    for _ in range(3):
        g.step(10)
        o.step(10)
        assert_same_state(g, o, f"{kind} n={n}")
        assert_same_lists(g, o)
    stats = []
    for pre in ("1", "0"):
        os.environ["SOIL_PAIRS_PRE"] = pre
        try:
            h = system.from_workload(ctx, w)
            h.step(30)
            c = h.counts()
            stats.append((c.npairs, c.filter_candidates, c.filter_rechecked))
            h.close()
        finally:
            del os.environ["SOIL_PAIRS_PRE"]
    assert stats[0] == stats[1]
    g.close()
