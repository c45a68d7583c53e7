"""Memory, pinned words and streams that a closed system leaves to the next
ones of its context: results do not depend on what was there, systems that
live side by side share nothing, and the accounting returns to zero."""
import numpy as np
import pytest

from helpers import assert_same_lists, assert_same_state, pair
from soil_b200 import abi, system, workloads as W

pytestmark = pytest.mark.gpu


def _w(seed, n, **kw):
    w = W.poly("reuse", seed, n, 0.45, 1e-4, 0, harmonic_k=1e3, **kw)
    w.vel *= 3.0
    return w


def test_systems_one_after_another_and_side_by_side(ctx):
    base = ctx.bytes_in_use()
    sizes = [40000, 300, 9000, 70001, 301, 12000]
    live = []
    for k, n in enumerate(sizes):
        g, o = pair(ctx, _w(240 + k, n, shear_rate=0.1 if k % 3 == 2 else 0.0))
        live.append((g, o))
        for a, b in live:  # the others go on between
            a.step(4)
            b.step(4)
        if len(live) > 2:
            a, b = live.pop(0)
            assert_same_state(a, b)
            assert_same_lists(a, b)
            a.close()
    for a, b in live:
        assert_same_state(a, b)
        assert_same_lists(a, b)
        a.close()
    assert ctx.bytes_in_use() == base


def test_a_tight_budget_takes_what_it_took(ctx):
    """The budget counts what systems hold: one system fits again and again,
    a second beside it does not, and a failed one leaves nothing behind."""
    w = _w(250, 20000)
    probe = system.from_workload(ctx, w)
    before = ctx.bytes_in_use()
    probe.step(3)
    probe.sync()
    need = ctx.bytes_in_use()
    assert need >= before
    probe.close()
    free = ctx.bytes_in_use()
    tight = system.Context(0, hbm_budget_bytes=(need - free) + (1 << 20))
    for _ in range(4):
        s = system.from_workload(tight, w)
        s.step(3)
        s.sync()
        with pytest.raises(abi.SoilError):
            t = system.from_workload(tight, w)
            t.step(1)
        s.step(2)
        assert np.isfinite(s.atoms(local_only=True)["pos"]).all()
        s.close()
        t = None
    assert tight.bytes_in_use() == 0
    tight.close()
