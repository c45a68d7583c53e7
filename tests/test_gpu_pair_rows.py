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
