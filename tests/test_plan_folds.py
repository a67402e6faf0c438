"""Which quantize steps a replay folds into the matvec behind them (q38b_plan.cu: merge_plan), without a device."""
import ctypes as C

import pytest

from qwengine_b200 import formats as F

FORMATS = ["Q4_K", "IQ3_XXS", "Q2_K", "IQ2_S"]      # with and without mma fragments


@pytest.fixture(scope="module")
def folds():
    from qwengine_b200 import build, load_library
    build.build()
    fn = load_library().q38b_debug_quantize_folds
    fn.argtypes = [C.c_uint32] + [C.c_int] * 6

    def run(name, nb, src_len, src_off=0, dst_off=-1, K=1024, M=512):
        rc = fn(F.get(name).type_id, nb, K, M, src_len, src_off, dst_off)
        assert rc in (0, 1)
        return bool(rc)
    return run


@pytest.mark.parametrize("name", FORMATS)
def test_columns_that_start_at_odd_floats_are_not_folded(folds, name):
    """The kernels read the floats 16 bytes at a time: with several columns the buffer's length is their distance."""
    for nb in (1, 2, 3, 4):
        assert folds(name, nb, 1024)
        assert folds(name, nb, 4096, src_off=1028)
        assert not folds(name, nb, 4096, src_off=1030)
        for extra in (1, 2, 3):
            assert folds(name, nb, 1024 + extra) == (nb == 1)
        assert folds(name, nb, 1028)
