"""How the tensor-core GEMM cuts a product into tiles (tg_ex_gemm_schedule; host code, no GPU needed)."""
import ctypes as C

import pytest

SMS = 148


def schedule(library, m, n, k, b_mn=False, out_fp32=False, ldc=None):
    plan = (C.c_int32 * 3)()
    b = (1, n) if b_mn else (k, 1)
    assert library.tg_ex_gemm_schedule(k, 1, *b, ldc or n, m, n, k, int(out_fp32), SMS, plan) == 0, library.tg_error()
    return tuple(plan)


# Measured us: the form that costs of aligned rows choose, and the fastest.
@pytest.mark.parametrize("m,n,k,b_mn,aligned_choice,fastest", [
    (46070, 552, 2272, True, (192, 1, 0), (256, 1, 1)),   # 146.7, 119.8
    (23263, 296, 1864, True, (192, 1, 0), (128, 1, 1)),   # 60.9, 47.3
    (33057, 728, 848, True, (192, 1, 0), (256, 1, 1)),    # 63.3, 50.5
    (51837, 440, 664, False, (256, 1, 0), (256, 1, 1)),   # 64.9, 53.9
    (51837, 664, 440, True, (192, 1, 0), (256, 1, 1)),    # 79.0, 58.4
    (63576, 288, 600, False, (192, 1, 0), (192, 1, 1)),   # 56.3, 45.1
    (9158, 3104, 440, False, (256, 1, 0), (256, 1, 1)),   # 43.2, 35.8
    (1425, 1480, 3536, True, (128, 1, 0), (128, 1, 1))])  # 23.3, 18.9
def test_rows_off_the_cache_lines_are_priced(library, m, n, k, b_mn, aligned_choice, fastest):
    assert schedule(library, m, n, k, b_mn) == fastest
    plan = (C.c_int32 * 3)()  # the same product with rows padded to whole cache lines
    pad = lambda x: (x + 63) // 64 * 64
    b = (1, pad(n)) if b_mn else (pad(k), 1)
    assert library.tg_ex_gemm_schedule(pad(k), 1, *b, pad(n), m, n, k, 0, SMS, plan) == 0
    assert tuple(plan) == aligned_choice


def test_alignment_has_no_say_in_how_often_k_is_cut(library):
    cut = 0
    for m in (16, 100, 260, 445, 1140, 5000):
        for n in range(72, 1500, 88):
            for k in range(520, 8000, 504):
                plan = (C.c_int32 * 3)()
                pad = lambda x: (x + 63) // 64 * 64
                assert library.tg_ex_gemm_schedule(pad(k), 1, pad(k), 1, pad(n), m, n, k, 0, SMS, plan) == 0
                assert schedule(library, m, n, k)[1] == plan[1]
                cut += plan[1] > 1
    assert cut > 100


def test_what_the_kernel_does_not_take_is_refused(library):
    plan = (C.c_int32 * 3)()
    for a_col, n, k in ((1, 60, 64), (1, 68, 64), (1, 64, 32), (2, 64, 64)):
        assert library.tg_ex_gemm_schedule(k, a_col, k, 1, n, 128, n, k, 0, SMS, plan) < 0
        assert b"outside the tensor-core" in library.tg_error()
