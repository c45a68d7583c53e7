"""The launch shape of the resident steps (soil_b200/csrc/steps_shape.cuh)."""
import ctypes as C

import pytest

from internal_hooks import build_internal

SMEM = 220 * 1024


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    lib = build_internal(tmp_path_factory.mktemp("hook"), "steps_shape_hook")
    lib.shape_of.argtypes = [C.c_uint64] * 3 + [C.c_uint32] * 2 + [C.POINTER(C.c_uint64)]

    def f(n, pairs, sms, ent=0, img=0):
        out = (C.c_uint64 * 6)()
        ok = lib.shape_of(n, pairs, sms, ent, img, out)
        return dict(zip(("group", "threads", "grid", "ent", "img", "smem"), out)) if ok else None
    return f


SIZES = [1, 63, 1000, 4736, 18944, 18945, 37888, 37889, 75776, 75777, 120001, 150000, 151552]


def room(p):
    return SMEM - (56 * p["threads"] if p["threads"] > 256 else 0)


@pytest.mark.parametrize("sms", [148, 132, 40])
@pytest.mark.parametrize("n", SIZES)
def test_the_system_fits_its_ctas(shape, n, sms):
    p = shape(n, 3 * n, sms)
    assert (p is not None) == (n <= 1024 * sms)
    if p:
        roots = p["threads"] // p["group"]
        assert p["grid"] <= sms and p["threads"] <= 1024 and p["threads"] % 32 == 0
        assert (p["grid"] - 1) * roots < n <= p["grid"] * roots
        assert p["ent"] % 8 == 0 and 44 * p["img"] + 5 * p["ent"] <= room(p)
        assert p["smem"] <= SMEM + 16


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("per_root", [2, 6, 12])
def test_lists_get_the_room_they_need_or_no_launch(shape, n, per_root):
    """Whatever a launch reported fits the next one, as long as it fits a CTA at
    all (up to the rounding of the entries to 8)."""
    first = shape(n, per_root * n, 148)
    roots, most = first["threads"] // first["group"], room(first)
    for img in (0, roots // 2, first["img"], first["img"] + 1, 2 * roots, 7 * roots, 26 * roots):
        left = (most - 44 * img) // 5
        for ent in (1, first["ent"], first["ent"] + 1, left // 2, left - 8, left + 1):
            if ent <= 0:
                continue
            p = shape(n, per_root * n, 148, ent, img)
            assert (p is not None) == (44 * img + 5 * ((ent + 7) // 8 * 8) <= most), (ent, img)
            if p:
                assert p["ent"] >= ent and p["img"] >= img
                assert 44 * p["img"] + 5 * p["ent"] <= most
