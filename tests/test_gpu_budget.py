"""A context's HBM budget bounds the device memory its systems hold, not only
the bytes their arrays ask for: many small systems, and one whose arrays grow
again and again.  A quarter more than the budget is allowed for what the pool
adds to each array."""
import ctypes as C

import numpy as np
import pytest

from internal_hooks import build_internal
from soil_b200 import abi, system, workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pool_used(tmp_path_factory):
    lib = build_internal(tmp_path_factory.mktemp("hook"), "ctx_hook")
    lib.ctx_pool_used.restype = C.c_uint64
    lib.ctx_pool_used.argtypes = [C.c_void_p]
    return lambda ctx: lib.ctx_pool_used(ctx.h)


def test_budget_bounds_many_small_systems(pool_used):
    budget = 96 << 20
    c = system.Context(0, hbm_budget_bytes=budget)
    w = W.poly("budget", 301, 200, 0.45, 1e-4, 0, harmonic_k=1e3)
    live = []
    with pytest.raises(abi.SoilError):
        for _ in range(500):
            s = system.from_workload(c, w)
            live.append(s)
            s.step(2)
    assert len(live) > 8
    assert pool_used(c) <= budget * 5 // 4
    while len(live) > 3:
        live.pop().close()
    live[0].sync()
    assert pool_used(c) <= c.bytes_in_use() * 5 // 4 + (1 << 20)
    s = system.from_workload(c, w)  # what closed systems held serves new ones
    s.step(2)
    for t in live + [s]:
        t.close()
    assert c.bytes_in_use() == 0
    c.close()


def test_budget_bounds_arrays_that_grow(pool_used):
    c = system.Context(0, hbm_budget_bytes=1 << 30)
    w = W.poly("budget-grow", 302, 60000, 0.45, 1e-4, 0, harmonic_k=1e3)
    s = system.System(c, w.box, w.cfg, w.dt)
    rc = s.register_column("radius", 1, abi.SOIL_COL_FORWARD)
    at, n = 0, 500
    while at < w.n:  # each part outgrows the capacity before it
        k = np.s_[at:min(at + n, w.n)]
        s.add_atoms(w.tag[k], w.pos[k], w.vel[k], w.mass[k], w.cutoff[k], columns=[w.radius[k]])
        at, n = k.stop, n + n // 2
    s.set_harmonic(w.harmonic_k, rc)
    s.setup()
    s.step(3)
    s.sync()
    assert pool_used(c) <= c.bytes_in_use() * 5 // 4 + (1 << 20)
    s.close()
    c.close()
