"""Row lengths the one-column kernel has a plan for (q38b_api.cu: plan_gemv1) on a 148-SM device with 227 KB of shared
memory a CTA, without a device: the header sets no limit, so what had a plan keeps one."""
import ctypes as C

import pytest

from qwengine_b200 import formats as F

# the first and the longest row lengths around the end of what fits; longer rows than any model's, but accepted
LONGEST = {"Q2_K": 144384, "IQ2_XXS": 137216, "IQ2_XS": 148480, "IQ2_S": 144384, "IQ1_S": 145408, "IQ1_M": 141312}
ALWAYS = 125952      # every length up to here


@pytest.fixture(scope="module")
def lib():
    from qwengine_b200 import build, load_library
    build.build()
    lib = load_library()
    lib.q38b_debug_gemv1_rows.argtypes = [C.c_uint32, C.c_int, C.c_int, C.c_size_t, C.c_int, C.c_int]
    return lib


@pytest.mark.parametrize("name", sorted(LONGEST))
@pytest.mark.parametrize("pad", [0, 16])
def test_long_rows_have_a_plan(lib, name, pad):
    f = F.get(name)
    for K in list(range(256, ALWAYS + 1, 256)) + [LONGEST[name]]:
        plan = lib.q38b_debug_gemv1_rows(f.type_id, K, 17408, f.row_bytes(K) + pad, 1, 1)
        assert plan // 100000 == 1, (name, K)


@pytest.mark.parametrize("name", sorted(F.ALL_FORMATS))
def test_columns_share_launches_at_every_length(lib, name):
    """Columns of the one-column kernel's arithmetic: up to four a launch where they fit, else three or two, never one alone
    beside others; the launches of a call take equal numbers or one less."""
    fn = lib.q38b_debug_gemv1_cols
    fn.argtypes = [C.c_uint32, C.c_int, C.c_int, C.c_size_t, C.c_int]
    f = F.get(name)
    for K in range(256, 17408 + 1, 256):
        for pad in (0, 16):
            for nb in range(1, 9):
                took, left = [], nb
                while left:
                    took.append(fn(f.type_id, K, 5120, f.row_bytes(K) + pad, left))
                    assert 1 <= took[-1] <= min(4, left)
                    left -= took[-1]
                assert max(took) - min(took) <= 1 and (nb == 1 or (nb == 3 and took == [2, 1]) or min(took) >= 2 or took == [2, 2, 1] or took == [2, 2, 2, 1]), (name, K, nb, took)
            if K <= 8192:
                assert fn(f.type_id, K, 5120, f.row_bytes(K), 4) == 4
