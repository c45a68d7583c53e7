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


# Atom counts on both sides of every launch shape: the lanes per root (8 up to
# 18,944 atoms, 4 to 37,888, 2 to 75,776, 1 to 151,552), full and ragged CTAs,
# and the first size past one launch.
@pytest.mark.parametrize("n", [40, 333, 4737, 18944, 18945, 37889, 75777, 151552, 151553])
@pytest.mark.parametrize("newton", [1, 0])
def test_resident_steps_match_oracle(ctx, n, newton):
    w = W.poly("resident", 160 + n % 5, n, 0.45, 1e-4, 0, harmonic_k=1e3, newton=newton)
    w.vel *= 6.0
    calls = [1, 2, 17, 1, 9] if n < 30000 else [1, 11]
    g = _stepped(ctx, w, "2", calls)
    o = oracle.from_workload(w)
    o.step(sum(calls))
    assert_same_state(g, o, f"n={n}")
    assert_same_lists(g, o)
    g.close()


@pytest.mark.parametrize("phi,n", [(0.45, 30), (0.45, 120), (2.5, 700), (6.0, 300)])
def test_resident_steps_many_images_and_entries(ctx, phi, n):
    """Boxes so small that a root has images on both sides of an axis (up to
    26), and packings so dense that rows hold dozens of entries."""
    w = W.poly("resident-dense", 171, n, phi, 1e-5, 0, harmonic_k=1e2)
    g = _stepped(ctx, w, "2", [1, 25])
    o = oracle.from_workload(w)
    o.step(26)
    assert_same_state(g, o, f"phi={phi} n={n}")
    assert_same_lists(g, o)
    g.close()


def test_resident_steps_crowded_corner(ctx):
    """One CTA's roots hold far more entries than the mean: the launch says so
    with nothing written, and the run goes on (more shared memory, then one
    launch per phase) with the same results."""
    w = W.poly("resident-crowd", 172, 9000, 0.30, 1e-6, 0, harmonic_k=1e1)
    w.pos[:1500] = 1.0 + w.pos[:1500] / w.L * 2.0
    g = _stepped(ctx, w, "2", [1, 6, 5])
    o = oracle.from_workload(w)
    o.step(12)
    assert_same_state(g, o)
    assert_same_lists(g, o)
    g.close()


# Stretches of one launch a step (systems past one resident launch): calls of
# every length around the two column sets they alternate between, ends before
# a periodic sort, checks that trip after odd and even numbers of steps, and
# axes without images.
@pytest.mark.parametrize("sort_every", [0, 3, 8])
@pytest.mark.parametrize("speed,open_axes", [(0.3, 0), (40.0, 0), (40.0, 1), (15.0, 2)])
def test_stretches_match_one_launch_per_phase(ctx, sort_every, speed, open_axes):
    w = W.poly("stretch", 181 + sort_every, 151777, 0.45, 1e-4, 0, harmonic_k=1e3,
               sort_every=sort_every)
    w.vel *= speed
    calls = [1, 2, 3, 1, 4, 5, 2, 30]

    def boundary(s):
        if open_axes:
            s.set_boundary([abi.SOIL_BOUNDARY_FIXED] * open_axes
                           + [abi.SOIL_BOUNDARY_PERIODIC] * (3 - open_axes))

    out = []
    for mode in ("2", "0"):
        os.environ["SOIL_RESIDENT_STEPS"] = mode
        try:
            g = system.System(ctx, w.box, w.cfg, w.dt)
            boundary(g)
            rc = g.register_column("radius", 1, abi.SOIL_COL_FORWARD)
            g.add_atoms(w.tag, w.pos, w.vel, w.mass, w.cutoff, columns=[w.radius])
            g.set_harmonic(w.harmonic_k, rc)
            g.setup()
            for n in calls:
                g.step(n)
        finally:
            del os.environ["SOIL_RESIDENT_STEPS"]
        out.append(g)
    assert_same_state(*out, f"sort_every={sort_every} speed={speed} open={open_axes}")
    assert_same_lists(*out)
    a, b = out[0].counts(), out[1].counts()
    assert (a.rebuilds, a.sorts) == (b.rebuilds, b.sorts)
    if speed == 40.0:
        assert a.rebuilds > 2
    for g in out:
        g.close()
