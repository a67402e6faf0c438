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


@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("nb", [1, 2, 4])
def test_a_matvec_that_writes_over_its_own_source_is_not_folded_into(folds, name, nb):
    """Every CTA of a folded launch reads the floats while others store their rows: the rows must not lie in them.  (On a
    device the unfolded order would be lost without a trace, so this is asked of the planner alone.)"""
    K, M = 1024, 512
    for dst_off, clear in [(0, False), (1020, False), (1023, False), (1024, True), (3584, True)]:
        assert folds(name, nb, 4096, 0, dst_off, K, M) == clear
    for dst_off, clear in [(0, True), (1536, True), (1540, False), (2560, False), (3071, False), (3072, True)]:
        assert folds(name, nb, 4096, 2048, dst_off, K, M) == clear


def test_rows_written_twice_do_not_share_a_launch():
    """The later of two matvecs that write the same rows wins; in one launch either could."""
    import numpy as np
    from qwengine_b200 import build, load_library
    build.build()
    fn = load_library().q38b_debug_merge_plan
    i32p = np.ctypeslib.ndpointer(np.int32, flags="C_CONTIGUOUS")
    fn.argtypes = [C.c_int, C.c_int, C.c_int, i32p, i32p]
    for nb in (1, 4):
        for off, at in [(0, 1), (508, 1), (512, 0), (-4, 1)]:      # 512 rows each, the first matvec's from float 4
            steps = np.array([(1, 4, 4), (1, 4, 4 + off)], np.int32)
            out = np.zeros(2, np.int32)
            fn(1, nb, 2, steps, out)
            assert out.tolist() == [0, at], (nb, off)
        # ... nor is a third matvec let into the first one's launch past a second that must come between
        out = np.zeros(3, np.int32)
        fn(1, nb, 3, np.array([(1, 4, 0), (1, 4, 0), (1, 4, 1024)], np.int32), out)
        assert out.tolist() == [0, 1, 1]
