"""Cuts that prefill_cut (q38b_prefill.cu) must not pick on a 148-SM device: each was measured slower, in us, than the one beside it.
One set of constants for all formats had picked them: the expanders of IQ4_XS take twice the time of Q4_K's."""
import ctypes as C

import pytest

from qwengine_b200 import formats as F


@pytest.fixture(scope="module")
def lib():
    from qwengine_b200 import build, load_library
    build.build()
    lib = load_library()
    lib.q38b_debug_prefill_plan.argtypes = [C.c_uint32, C.c_int, C.c_int, C.c_int, C.POINTER(C.c_int)]
    return lib


def cut(lib, name, M, K, B):
    out = (C.c_int * 4)()
    assert lib.q38b_debug_prefill_plan(F.get(name).type_id, K, M, B, out) == 0
    return tuple(out[:3])      # token tiles, tokens a tile, CTAs that share K


@pytest.mark.parametrize("name,M,K,B,slow,us,fast,fast_us", [
    ("IQ4_XS", 5120, 17408, 1024, (3, 384, 1), 198.3, (2, 512, 3), 186.7),
    ("IQ3_XXS", 5120, 17408, 1024, (3, 384, 1), 188.1, (2, 512, 3), 178.2),
    ("IQ2_XS", 5120, 17408, 1024, (3, 384, 1), 181.9, (2, 512, 3), 174.7),
    ("IQ3_XXS", 2816, 9728, 768, (2, 384, 3), 54.3, (3, 256, 2), 46.1),
    ("IQ2_XS", 4096, 4096, 512, (1, 512, 4), 29.7, (2, 256, 2), 25.6),
    ("Q4_K", 5120, 17408, 1024, (3, 384, 1), 164.9, (5, 208, 2), 149.1),
])
def test_measured_cuts(lib, name, M, K, B, slow, us, fast, fast_us):
    got = cut(lib, name, M, K, B)
    assert got != slow, (us, fast_us)
    assert got == fast


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
def test_every_call_has_a_cut(lib, name):
    for M in (1, 128, 129, 5120, 248320):
        for K in (256, 512, 5120, 17408):
            for B in (1, 16, 17, 256, 257, 512, 513, 2500):
                tiles, tile, splits = cut(lib, name, M, K, B)
                assert tiles * tile >= B and (tiles - 1) * tile < B and 1 <= splits <= min(8, K // 256)
