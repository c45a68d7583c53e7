"""Which form light steps take, seen by the kernel launches they issue."""
import ctypes as C
import os

import pytest

import oracle
from helpers import assert_same_lists, assert_same_state
from internal_hooks import build_internal
from soil_b200 import abi, system, workloads as W

pytestmark = pytest.mark.gpu


def _launches(g, n):
    lib = abi.load_library()
    l0 = lib.soil_kernel_launches()
    g.step(n)
    return lib.soil_kernel_launches() - l0


@pytest.fixture(scope="module")
def hook(tmp_path_factory):
    lib = build_internal(tmp_path_factory.mktemp("hook"), "ctx_hook")
    lib.ctx_get_sms.restype = C.c_uint64
    lib.ctx_get_sms.argtypes = [C.c_void_p]
    lib.ctx_set_sms.argtypes = [C.c_void_p, C.c_uint64]
    return lib


# 37 SMs hold up to 37,888 roots: 9,000 (4 lanes each) and 37,888 (1) take the
# resident launch, 37,889 one launch a step.  A shape for 40,000 SMs asks for
# more CTAs than any device holds at once: the launch is refused, and small and
# large systems go on without it.
@pytest.mark.parametrize("sms,n,resident", [(37, 9000, True), (37, 37888, True), (37, 37889, False),
                                            (40000, 37800, False), (40000, 60000, False)])
def test_resident_launch_is_shaped_for_the_device(hook, sms, n, resident):
    import torch
    c = system.Context(0)
    assert hook.ctx_get_sms(c.h) == torch.cuda.get_device_properties(0).multi_processor_count
    hook.ctx_set_sms(c.h, sms)
    w = W.poly("forms-sms", 322, n, 0.45, 1e-5, 0, harmonic_k=1e3)
    g, o = system.from_workload(c, w), oracle.from_workload(w)
    g.step(1)
    launches = _launches(g, 12)
    assert g.counts().rebuilds == 1
    assert launches <= 2 if resident else launches >= 12, launches
    o.step(13)
    assert_same_state(g, o)
    assert_same_lists(g, o)
    g.close()
    c.close()


def _crowded(n, crowd, side):
    """A packing with `crowd` more atoms in a cube of `side` at its centre."""
    w = W.poly("forms", 320, n, 0.45, 1e-7, 0, harmonic_k=1e1)
    w.pos[:crowd] = 0.5 * w.L + (w.pos[:crowd] / w.L - 0.5) * side
    return w


# (9,000: 8 lanes per root, 64 roots a CTA; 150,000: 1 lane, 1,024 roots, where
# shared memory is shortest)
@pytest.mark.parametrize("n,crowd,side", [(9000, 200, 2.5), (150000, 300, 3.0)])
def test_lists_that_need_more_room_stay_resident(ctx, n, crowd, side):
    w = _crowded(n, crowd, side)
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    g.step(1)
    first = _launches(g, 12)  # the launch that did not fit, the one that did, the last half-kick
    again = _launches(g, 12)
    assert g.counts().rebuilds == 1
    o.step(25)
    assert_same_state(g, o)
    assert_same_lists(g, o)
    assert first <= 4 and again <= 2, (first, again)
    g.close()


def test_lists_that_never_fit_step_by_launches(ctx):
    w = _crowded(9000, 3000, 2.0)
    g, o = system.from_workload(ctx, w), oracle.from_workload(w)
    g.step(1)
    assert _launches(g, 12) >= 24 and _launches(g, 12) >= 24
    assert g.counts().rebuilds == 1
    o.step(25)
    assert_same_state(g, o)
    assert_same_lists(g, o)
    g.close()


@pytest.mark.parametrize("force,resident", [("csr", True), ("walk", False), ("tiles4", False),
                                            ("tiles2", False), ("gather", False)])
def test_light_steps_run_the_kernel_soil_force_names(ctx, force, resident):
    """Only the CSR walk has a resident form; the others launch in every step."""
    w = W.poly("forms-force", 321, 4000, 0.45, 1e-5, 0, harmonic_k=1e3)
    o = oracle.from_workload(w)
    old = os.environ.get("SOIL_FORCE")
    os.environ["SOIL_FORCE"] = force
    try:
        g = system.from_workload(ctx, w)
        g.step(1)
        launches = _launches(g, 40)
    finally:
        if old is None:
            del os.environ["SOIL_FORCE"]
        else:
            os.environ["SOIL_FORCE"] = old
    assert g.counts().rebuilds == 1
    assert launches <= 4 if resident else launches >= 80, launches
    o.step(41)
    assert_same_state(g, o, force)
    g.close()


@pytest.mark.parametrize("force", ["walk", "tiles2", "gather"])
@pytest.mark.parametrize("newton,reverse", [(1, 0), (1, 1), (0, 0)])
def test_named_kernels_step_alike_with_and_without_the_host(ctx, force, newton, reverse):
    """Light steps whose check's answer the host reads while forward comm runs
    give the bits of one launch per phase, #[reverse] columns included."""
    w = W.poly("forms-named", 323, 6000, 0.5, 1e-3, 0, harmonic_k=1e3, newton=newton)
    w.vel *= 2.0
    out = []
    keys = ("SOIL_FORCE", "SOIL_RESIDENT_STEPS")
    old = {k: os.environ.get(k) for k in keys}
    try:
        for mode in ("2", "0"):
            os.environ.update(dict(zip(keys, (force, mode))))
            g = system.System(ctx, w.box, w.cfg, w.dt)
            rc = g.register_column("radius", 1, abi.SOIL_COL_FORWARD)
            cols = [w.radius]
            if reverse:
                g.register_column("acc", 1, abi.SOIL_COL_REVERSE)
                cols.append(1.0 + w.pos[:, 0])
            g.add_atoms(w.tag, w.pos, w.vel, w.mass, w.cutoff, columns=cols)
            g.set_harmonic(w.harmonic_k, rc)
            g.setup()
            for n in (1, 2, 1, 25):
                g.step(n)
            out.append(g)
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v
    assert_same_state(*out, force)
    assert_same_lists(*out)
    assert 2 < out[0].counts().rebuilds < 29
    for g in out:
        g.close()
