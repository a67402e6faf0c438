"""How the several-column kernel divides a row (q38b_gemvn.cu: plan_gemv, q38b_cols_take), without a device: the choices that were
measured slow stay out.  Whole tiles in one copy where many of their rows meet on a bank (17408 x 5120 Q8_0, seven columns, 39.1 us
against 27.0), a handful of warps, all columns at once where a long row's activations
leave two small stages for a few warps (5120 x 17408 IQ3_XXS, per-32, eight columns 164 us against 69 as four and four)."""
import ctypes as C

import pytest

from qwengine_b200 import formats as F

ONE_COLUMN_BITS = ("Q2_K", "IQ2_XXS", "IQ2_XS", "IQ2_S", "IQ1_S", "IQ1_M")


@pytest.fixture(scope="module")
def lib():
    from qwengine_b200 import build, load_library
    build.build()
    lib = load_library()
    lib.q38b_debug_gemvn_plan.argtypes = [C.c_uint32, C.c_int, C.c_int, C.c_size_t, C.c_int, C.c_int, C.POINTER(C.c_int)]
    lib.q38b_debug_gemvn_take.argtypes = [C.c_uint32, C.c_int, C.c_int, C.c_size_t, C.c_int, C.c_int]
    return lib


def plan(lib, f, K, M, nb, a32, pad=0):
    out = (C.c_int * 6)()
    rc = lib.q38b_debug_gemvn_plan(f.type_id, K, M, f.row_bytes(K) + pad, nb, a32, out)
    return dict(zip(("kw", "groups", "chunk", "stages", "one_copy", "rating"), out)) if rc == 0 else None


# bytes of a lane's main load, distance between the four lanes of a row, rows served together
LOADS = {"Q4_K": (8, 8, 4), "Q5_K": (8, 8, 4), "Q8_0": (2, 8, 8), "IQ4_XS": (4, 4, 8), "Q2_K": (4, 4, 8), "Q6_K": (2, 4, 8), "IQ3_XXS": (2, 2, 8),
         "IQ3_S": (2, 2, 8), "IQ2_XS": (2, 2, 8)}


def most_words_of_a_bank(name, pitch):
    size, step, rows = LOADS.get(name, (1, 1, 8))
    banks = {}
    for g in range(rows):
        for t in range(4):
            for b in range(0, size, 4):
                w = (g * pitch + t * step + b) // 4
                banks.setdefault(w % 32, set()).add(w)
    return max(len(v) for v in banks.values())


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
@pytest.mark.parametrize("a32", [0, 1])
def test_rows_up_to_8192(lib, name, a32):
    f = F.get(name)
    for K in range(1024, 8192 + 1, 256):
        for nb in range(2, 9):
            for pad in (0, 16):
                p = plan(lib, f, K, 17408, nb, a32, pad)
                assert p, (name, K, nb)
                assert not (p["one_copy"] and pad), (name, K, nb, p)
                assert p["stages"] >= 2 * p["groups"]
                assert not p["one_copy"] or f.row_bytes(K) <= 1536 or most_words_of_a_bank(name, f.row_bytes(K)) <= 3, (name, K, nb, p)
                assert p["kw"] * p["groups"] >= 7, (name, K, nb, p)
                assert lib.q38b_debug_gemvn_take(f.type_id, K, 17408, f.row_bytes(K) + pad, nb, a32) == (0 if a32 and name == "Q6_K" else nb)


@pytest.mark.parametrize("nb", range(2, 9))
def test_rows_that_meet_on_banks_are_copied_apart(lib, nb):
    for K in (5120, 6144, 7168):
        assert plan(lib, F.get("Q8_0"), K, 17408, nb, 0)["one_copy"] == 0


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
@pytest.mark.parametrize("a32", [0, 1])
def test_long_rows_never_take_columns_that_starve_the_ring(lib, name, a32):
    f = F.get(name)
    if a32 and name == "Q6_K":
        return
    for K in range(8448, 32768 + 1, 1024):
        for left in range(2, 9):
            n = lib.q38b_debug_gemvn_take(f.type_id, K, 5120, f.row_bytes(K), left, a32)
            assert 1 <= n <= left
            if n > 1:
                p, h = plan(lib, f, K, 5120, n, a32), plan(lib, f, K, 5120, (n + 1) // 2, a32)
                assert p["rating"] >= min(250, 0.2 * h["rating"]) - 1, (name, K, left, p, h)
    if a32 and name == "IQ3_XXS":
        assert lib.q38b_debug_gemvn_take(f.type_id, 17408, 5120, f.row_bytes(17408), 8, 1) == 4
