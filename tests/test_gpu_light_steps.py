"""Stretches of steps that keep their lists, at the sizes where their kernels
can go wrong: bit-identical to one launch per phase (SOIL_RESIDENT_STEPS=0)
and to the CPU oracle, whatever the atom count, the call lengths and where
the displacement check trips."""
import os

import pytest

import oracle
from helpers import assert_same_lists, assert_same_state
from soil_b200 import abi, system, workloads as W

pytestmark = pytest.mark.gpu


def _stepped(ctx, w, mode, calls, prepare=None):
    old = os.environ.get("SOIL_RESIDENT_STEPS")
    os.environ["SOIL_RESIDENT_STEPS"] = mode
    try:
        g = system.from_workload(ctx, w)
        if prepare:
            prepare(g)
        for n in calls:
            g.step(n)
        return g
    finally:
        if old is None:
            del os.environ["SOIL_RESIDENT_STEPS"]
        else:
            os.environ["SOIL_RESIDENT_STEPS"] = old


# Atom counts around the thread, block and one-wave edges of the two launches.
@pytest.mark.parametrize("n", [64, 255, 257, 4099, 300007])
@pytest.mark.parametrize("speed", [0.0, 1.0, 40.0])
def test_free_flight_matches_oracle(ctx, n, speed):
    w = W.mono("flight", 140 + n % 7, n, 0.30, 1e-3, 0)
    w.vel *= speed
    calls = [1, 2, 29, 1, 12] if n < 100000 else [1, 14]
    g = _stepped(ctx, w, "2", calls)
    o = oracle.from_workload(w)
    o.step(sum(calls))
    assert_same_state(g, o, f"n={n} speed={speed}")
    assert_same_lists(g, o)
    if speed == 40.0:
        assert g.counts().rebuilds > 2
    g.close()


@pytest.mark.parametrize("sort_every", [0, 3, 7])
def test_free_flight_ends_before_a_periodic_sort(ctx, sort_every):
    w = W.poly("flight-sort", 151, 3001, 0.35, 1e-3, 0, sort_every=sort_every)
    g = _stepped(ctx, w, "2", [40])
    o = oracle.from_workload(w)
    o.step(40)
    assert_same_state(g, o)
    assert_same_lists(g, o)
    g.close()


def test_free_flight_takes_up_the_forces_of_a_removed_consumer(ctx):
    """The first pass of a flight still applies the forces the columns hold."""
    w = W.poly("flight-left", 152, 2000, 0.5, 1e-4, 0, harmonic_k=1e3)

    def drop(g):
        g.step(5)
        g.set_harmonic(0.0, -1)

    a = _stepped(ctx, w, "2", [30], drop)
    b = _stepped(ctx, w, "0", [30], drop)
    assert_same_state(a, b)
    assert a.counts().comm_state == abi.SOIL_COMMUNICATE_ONLY
    a.close()
    b.close()
