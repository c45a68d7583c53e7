"""The places of a system's arrays in its slabs (soil_b200/csrc/arena.cuh)."""
import ctypes as C
import random

import pytest

from internal_hooks import build_internal

MB = 1 << 20


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    lib = build_internal(tmp_path_factory.mktemp("hook"), "arena_hook")
    u64, p = C.c_uint64, C.c_void_p
    for name, res, args in (("arena_new", p, []), ("arena_delete", None, [p]),
                            ("arena_take", u64, [p, u64]), ("arena_give", None, [p, u64, u64]),
                            ("arena_next_slab", u64, [p, u64]),
                            ("arena_add", u64, [p, u64, u64, u64]), ("arena_lost", u64, [p, u64]),
                            ("kept_new", p, []), ("kept_delete", None, [p]),
                            ("kept_give", C.c_int, [p, u64, u64]),
                            ("kept_take", u64, [p, u64, u64]), ("kept_bytes", u64, [p])):
        f = getattr(lib, name)
        f.restype, f.argtypes = res, args
    return lib


@pytest.mark.parametrize("seed", range(4))
def test_arrays_never_overlap_and_nothing_is_lost(lib, seed):
    """Arrays that grow and go: their places are disjoint and inside slabs, and
    every byte of a slab is an array's, free, or not handed out yet."""
    rng = random.Random(seed)
    a = lib.arena_new()
    slabs, live, base = [], [], 1 << 40
    for _ in range(3000):
        if live and rng.random() < 0.45:
            p, n = live.pop(rng.randrange(len(live)))
            lib.arena_give(a, p, n)
            n = n * 5 // 4 // 256 * 256 + 256  # an array that grows
        else:
            n = 256 * int(2 ** rng.uniform(0, 15))
        n = min(n, 8 * MB)
        p = lib.arena_take(a, n)
        if not p:
            size = lib.arena_next_slab(a, n)
            assert max(n, MB) <= size <= max(n, 32 * MB)
            p = lib.arena_add(a, base, size, n)
            slabs.append((base, size))
            base += size + MB
        live.append((p, n))
        assert lib.arena_lost(a, sum(k for _, k in live)) == 0
    at = 0
    for p, n in sorted(live):
        assert p % 256 == 0 and p >= at
        at = p + n
        assert any(b <= p and p + n <= b + s for b, s in slabs)
    lib.arena_delete(a)


def test_kept_slabs_go_to_systems_of_their_size(lib):
    """A kept slab serves a system that wants at least half of it, smaller ones
    when there is none; more than 512 MB are not kept."""
    k = lib.kept_new()
    for n in (32, 2, 1, 1):
        assert lib.kept_give(k, n * MB, n * MB)
    assert lib.kept_take(k, 1 * MB, 4096) == 1 * MB
    assert lib.kept_take(k, 1 * MB, 4096) == 1 * MB
    assert lib.kept_take(k, 1 * MB, 4096) == 2 * MB
    assert lib.kept_take(k, 1 * MB, 4096) == 0  # only the 32 MB slab is left
    assert lib.kept_take(k, 15 * MB, 4096) == 0
    assert lib.kept_give(k, MB, MB)
    assert lib.kept_take(k, 8 * MB, 8 * MB) == 0
    assert lib.kept_take(k, 8 * MB, 4096) == 1 * MB  # none of 8 to 16: the smaller one
    assert lib.kept_take(k, 16 * MB, 16 * MB) == 32 * MB
    assert lib.kept_bytes(k) == 0
    for _ in range(16):
        assert lib.kept_give(k, 32 * MB, 32 * MB)
    assert not lib.kept_give(k, MB, MB)
    assert lib.kept_bytes(k) == 512 * MB
    lib.kept_delete(k)
