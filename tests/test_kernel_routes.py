"""Which kernel a call takes, where a rule on its sizes decides, and what is refused before anything is launched (no GPU)."""
import ctypes

import pytest

from hymt2sharp_b200.kernels import ops


@pytest.mark.parametrize("rows, vocab, filters, draw", [
    (8, 120818, 8, 8), (64, 120818, 8, 8), (65, 120818, 1, 8), (100, 120818, 1, 8), (101, 120818, 1, 1), (148, 300000, 8, 1), (64, 32768, 8, 8),
    (256, 32768, 1, 8), (256, 65536, 1, 8), (256, 300, 1, 1), (1, 300, 1, 1), (8, 5000, 1, 1), (8, 12000, 8, 1), (40, 16384, 8, 1), (41, 16384, 1, 1),
    (33, 20000, 8, 1), (32, 20000, 8, 8), (1, 408576, 8, 8), (1, 408577, 8, 1), (2 ** 31 - 1, 120818, 1, 1)])
def test_rows_are_filtered_and_drawn_by_one_block_where_a_cluster_would_be_slower(rows, vocab, filters, draw):
    assert (ops.filter_blocks(rows, vocab), ops.sample_blocks(rows, vocab)) == (filters, draw)


@pytest.mark.parametrize("rows, vocab, resident", [(1, 120818, 1), (14, 120818, 1), (15, 120818, 2), (64, 120818, 2), (64, 5000, 1), (148, 5000, 1), (149, 5000, 2)])
def test_blocks_of_the_filters_share_an_sm_where_they_would_wait_for_one(rows, vocab, resident):
    assert ops.filter_resident(rows, vocab) == resident


@pytest.mark.parametrize("rows, columns, epilogue, narrow, kernel", [
    (129, 2048, 0, True, "64x64 short"), (300, 1000, 0, True, "64x64 short"), (600, 500, 0, True, "64x64 short"), (1, 8192, 0, True, "64x64 short"),
    (129, 4096, 2, True, "64x64"), (64, 9472, 0, True, "64x64 short"), (64, 9473, 0, True, "64x128"), (531, 6144, 2, True, "64x128"),
    (531, 3072, 0, False, "64x64"), (531, 6144, 2, False, "64x128"), (129, 2048, 0, False, "64x64"), (65, 130, 0, False, "32x64")])
def test_tiles_of_products_on_cuda_cores(rows, columns, epilogue, narrow, kernel):
    assert ops.gemm_simt_route(rows, columns, epilogue, narrow=narrow) == kernel


@pytest.mark.parametrize("rows, widest, widest_gated", [(1, 10 ** 6, 10 ** 6), (8, 10 ** 6, 10 ** 6), (9, 20480, 10 ** 6), (16, 20480, 10 ** 6), (17, 9472, 9472),
                                                        (32, 9472, 9472), (33, 4736, 2368), (64, 4736, 2368), (65, 0, 0)])
def test_few_rows_stream_their_weights_as_far_as_that_is_faster(rows, widest, widest_gated):
    for epilogue, last in ((ops.EPILOGUE_STORE, widest), (ops.EPILOGUE_ACCUMULATE, widest), (ops.EPILOGUE_SWIGLU, widest_gated)):
        if last:
            assert ops.gemm_simt_route(rows, last, epilogue) == "rows"
        if last < 10 ** 6:
            assert ops.gemm_simt_route(rows, last + 1, epilogue) != "rows"
        assert ops.gemm_simt_route(rows, 64, epilogue, aligned=False) != "rows" and ops.gemm_simt_route(rows, 64, epilogue, batch=2) != "rows"
        assert ops.gemm_simt_route(rows, 64, epilogue, narrow=True) != "rows"


@pytest.mark.parametrize("tokens, heads, d, rows", [(531, 16, 128, 32), (1183, 16, 128, 32), (1184, 16, 128, 64), (4096, 16, 96, 64), (4096, 16, 88, 32), (4096, 16, 64, 32),
                                                    (4096, 16, 24, 32), (4096, 16, 136, 32), (18944, 1, 128, 64)])
def test_rows_a_block_of_32_bit_prompt_attention(tokens, heads, d, rows):
    assert ops.attention_prompt_rows(tokens, heads, d) == rows


@pytest.mark.parametrize("lda, ldw, ldc", [(2044, 2048, 1024), (0, 2048, 1024), (2048, 2044, 1024), (2048, 0, 1024), (2048, 2048, 1023), (2048, 2048, 0)])
def test_float32_products_refuse_rows_that_overlap(lda, ldw, ldc):
    """As the CUDA-core product does: such rows of C would be written by several at once."""
    lib, at = ops._lib(), 1 << 20          # (an address that nothing gets to read)
    for name, call in (("gemm_f32_tc", lambda: lib.hymt2_gemm_f32_tc(at, at, at, 8, 1024, 2048, lda, ldw, ldc, 0, None, 0, at, None, 0, 0.0, 1.0, None)),
                       ("gemm", lambda: lib.hymt2_gemm_simt(ctypes.c_void_p(at), 0, ctypes.c_void_p(at), 0, ctypes.c_void_p(at), 0, 8, 1024, 2048,
                                                            ctypes.c_long(lda), ctypes.c_long(ldw), ctypes.c_long(ldc), 0, 0, ctypes.c_float(0),
                                                            ctypes.c_float(1), None, None))):
        assert call() == -1
        assert "leading dimension is smaller than its row" in lib.hymt2_last_error().decode(), name
