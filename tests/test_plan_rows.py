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
    """Columns of the one-column kernel's arithmetic: a launch takes the most that fit, four or at long rows of some formats
    three or two, never one of several."""
    fn = lib.q38b_debug_gemv1_cols
    fn.argtypes = [C.c_uint32, C.c_int, C.c_int, C.c_size_t, C.c_int]
    f = F.get(name)
    for K in range(256, 17408 + 1, 256):
        for pad in (0, 16):
            took = [fn(f.type_id, K, 5120, f.row_bytes(K) + pad, left) for left in range(1, 9)]
            assert took[0] == 1 and took[1] == 2 and took[4:] == [took[3], took[2], took[3], took[3]], (name, K, took)
            assert 2 <= took[2] <= took[3] <= 4, (name, K, took)
            if K <= 8192:
                assert took[2:4] == [3, 4]
