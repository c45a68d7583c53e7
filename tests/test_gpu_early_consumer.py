"""The consumer queued behind a rebuild before the host knows the sizes, when
the ghosts or the pairs of that rebuild outgrow their arrays: it must not run
(its lists are not all written), the build is repeated, and each phase is timed
once.  And light steps with phase timers on, where a check trips."""
import numpy as np
import pytest

import oracle
from helpers import assert_same_lists, assert_same_state
from soil_b200 import abi, system, workloads as W

pytestmark = pytest.mark.gpu
T = {name: k for k, name in enumerate(abi.TIMER_NAMES)}


def _moving(w, between, target):
    """Atoms anywhere at first, at `between` after one step, at `target` after two."""
    w.vel[:] = (target - between) / w.dt
    w.pos[:] = (2.0 * between - target) % w.L
    return w


def _to_the_faces(n, newton):
    """A dilute gas that ends mostly on a grid just inside the six faces: many
    more ghosts, few pairs (the pair total does not outgrow its arrays)."""
    w = W.poly("faces", 310, n, 0.02, 1e-4, 0, harmonic_k=1.0, newton=newton)
    rng = np.random.default_rng(310)
    m = int(w.L / 1.5)
    g = (np.arange(m) + 0.5) * (w.L / m)
    u, v = (a.ravel() for a in np.meshgrid(g, g, indexing="ij"))
    half = 0.5 * w.L / m
    faces = []
    for d in range(3):
        for side in (0, 1):
            p = np.empty((m * m, 3))
            p[:, (d + 1) % 3] = (u + side * half) % w.L
            p[:, (d + 2) % 3] = (v + side * half) % w.L
            p[:, d] = 0.55 if side == 0 else w.L - 0.55
            faces.append(p)
    grid = np.concatenate(faces)
    grid = grid[rng.permutation(len(grid))][:n * 9 // 10]
    target = rng.uniform(0.0, w.L, (n, 3))
    target[:len(grid)] = grid
    return _moving(w, rng.uniform(0.0, w.L, (n, 3)), target)


def _to_the_middle(n, newton):
    """A gas that ends in the middle eighth of the box: no ghosts, eight times
    the pairs."""
    w = W.poly("middle", 312, n, 0.05, 1e-4, 0, harmonic_k=1.0, newton=newton)
    rng = np.random.default_rng(312)
    return _moving(w, rng.uniform(0.0, w.L, (n, 3)), rng.uniform(0.25, 0.75, (n, 3)) * w.L)


# 8 lanes per root up to 37,888 roots, one thread per root (and 8 lanes for the
# roots with several images) above
@pytest.mark.parametrize("n", [20000, 40000])
@pytest.mark.parametrize("newton", [1, 0])
def test_ghosts_outgrow_their_arrays_on_a_later_rebuild(ctx, n, newton):
    w = _to_the_faces(n, newton)
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    g.step(1)
    o.step(1)
    room, pairs = g.view().stride, g.counts().npairs
    g.set_timing((1 << abi.SOIL_NUM_TIMERS) - 1)
    g.step(1)
    o.step(1)
    c = g.counts()
    assert c.nlocal + c.nghost > room and g.view().stride > room
    assert 0 < c.npairs <= 2 * pairs  # the pair arrays had room: only the ghosts had not
    assert_same_state(g, o, f"n={n} newton={newton}")
    assert_same_lists(g, o)
    _, _, iv = g.get_timing()
    assert iv[T["force"]] == 1 and iv[T["neighbor"]] == 1
    g.step(2)
    o.step(2)
    assert_same_state(g, o)
    g.close()


@pytest.mark.parametrize("n", [20000, 40000])
@pytest.mark.parametrize("newton", [1, 0])
def test_pairs_outgrow_their_arrays_on_a_later_rebuild(ctx, n, newton):
    w = _to_the_middle(n, newton)
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    g.step(1)
    o.step(1)
    pairs = g.counts().npairs
    g.set_timing((1 << abi.SOIL_NUM_TIMERS) - 1)
    g.step(1)
    o.step(1)
    assert g.counts().npairs > 4 * pairs
    assert_same_state(g, o, f"n={n} newton={newton}")
    assert_same_lists(g, o)
    _, _, iv = g.get_timing()
    assert iv[T["force"]] == 1 and iv[T["neighbor"]] == 1
    g.close()


@pytest.mark.parametrize("newton", [1, 0])
@pytest.mark.parametrize("n", [5000, 45000])
def test_timed_light_steps_drop_the_phases_of_a_tripped_check(ctx, n, newton):
    w = W.poly("timed", 311, n, 0.5, 1e-3, 0, harmonic_k=1e3, newton=newton)
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    g.step(1)
    o.step(1)
    g.set_timing((1 << abi.SOIL_NUM_TIMERS) - 1)
    built, steps = g.counts().rebuilds, 0
    while g.counts().rebuilds < built + 3:
        g.step(20)
        o.step(20)
        steps += 20
    assert_same_state(g, o, f"n={n}")
    assert_same_lists(g, o)
    _, _, iv = g.get_timing()
    rebuilds = g.counts().rebuilds - built
    assert rebuilds < steps
    assert iv[T["integrate"]] == iv[T["force"]] == steps
    # a rebuild step's forward phase is empty but timed; a dropped one is not
    assert iv[T["forward"]] == steps
    assert iv[T["neighbor"]] == iv[T["borders"]] == rebuilds
    g.close()
