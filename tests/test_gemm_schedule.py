"""How the tensor-core GEMM cuts a product into tiles (tg_ex_gemm_schedule; host code, no GPU needed)."""
import ctypes as C

import pytest

SMS = 148


def schedule(library, m, n, k, b_mn=False, batch=1, beside_others=False, pitch=lambda x: x):
    """(tile columns, K splits, CTA pair, half an SM)"""
    plan = (C.c_int32 * 4)()
    b = (1, pitch(n)) if b_mn else (pitch(k), 1)
    assert library.tg_ex_gemm_schedule(pitch(k), 1, *b, pitch(n), m, n, k, batch, 0, int(beside_others), SMS, plan) == 0, \
        library.tg_error()
    return tuple(plan)


def whole_lines(elements):
    return (elements + 63) // 64 * 64


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
    assert schedule(library, m, n, k, b_mn)[:3] == fastest
    assert schedule(library, m, n, k, b_mn, pitch=whole_lines)[:3] == aligned_choice


# Measured us: the form that the costs for any N choose, and the fastest.
@pytest.mark.parametrize("m,n,k,b_mn,fastest", [
    (32768, 768, 768, False, (192, 1, 1)),    # 41.0, 34.6
    (32768, 768, 768, True, (256, 1, 1)),     # 40.9, 36.2
    (8192, 1536, 384, False, (256, 1, 1)),    # 12.4, 10.7
    (4096, 3072, 768, False, (256, 1, 1))])   # 18.0, 15.9
def test_outputs_of_whole_blocks_have_costs_of_their_own(library, m, n, k, b_mn, fastest):
    assert schedule(library, m, n, k, b_mn)[:3] == fastest


# Measured us: single tiles of 256 columns, and pairs; the last two keep A in L2.
@pytest.mark.parametrize("m,n,k,b_mn,fastest", [
    (17871, 256, 3456, False, (256, 1, 1)),   # 36.6, 30.4
    (13865, 256, 3520, False, (256, 1, 1)),   # 29.8, 26.1
    (52096, 1024, 3072, True, (256, 1, 1)),   # 238.1, 221.7
    (32768, 1024, 4096, False, (256, 1, 1)),  # 201.2, 180.7
    (18719, 256, 960, False, (256, 1, 0)),    # 13.8, 14.6
    (18078, 256, 1024, False, (256, 1, 0))])  # 13.2, 14.1
def test_a_product_whose_input_streams_from_memory_takes_pairs(library, m, n, k, b_mn, fastest):
    assert schedule(library, m, n, k, b_mn)[:3] == fastest


def test_alignment_has_no_say_in_how_often_k_is_cut(library):
    cut = 0
    for m in (16, 100, 260, 445, 1140, 5000):
        for n in range(72, 1500, 88):
            for k in range(520, 8000, 504):
                splits = schedule(library, m, n, k)[1]
                assert splits == schedule(library, m, n, k, pitch=whole_lines)[1]
                cut += splits > 1
    assert cut > 100


@pytest.mark.parametrize("depth,width", [(6, 384), (3, 320), (2, 1024), (4, 768)])  # the last two: a rank's share of 16 and 12 layers
def test_half_an_sm_only_beside_others(library, depth, width):
    """The products of Muon's square and wide matrices: A = X X^T, A A, and B X.  A chain that has the GPU to itself (data
    parallelism, a profiled engine, a large model) keeps the deep ring."""
    halves = 0
    for n in (width, 3 * width, 4 * width):
        for m, columns, k, b_mn in ((width, width, n, False), (width, width, width, True), (width, n, width, True)):
            alone = schedule(library, m, columns, k, b_mn, depth)
            beside = schedule(library, m, columns, k, b_mn, depth, True)
            assert alone[3] == 0 and beside[:3] == alone[:3]
            assert not beside[3] or (beside[0] <= 128 and not beside[2])
            halves += beside[3]
    assert halves >= 6
    assert schedule(library, width, width, width, True, 1, True)[3] == 0  # one matrix is no batch


def test_what_the_kernel_does_not_take_is_refused(library):
    plan = (C.c_int32 * 4)()
    for a_col, n, k in ((1, 60, 64), (1, 68, 64), (1, 64, 32), (2, 64, 64)):
        assert library.tg_ex_gemm_schedule(k, a_col, k, 1, n, 128, n, k, 1, 0, 0, SMS, plan) < 0
        assert b"outside the tensor-core" in library.tg_error()
