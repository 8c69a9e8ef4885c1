"""Which form a product takes (CPU): the lines that measurement drew, on 148 SMs, for products of the presets and at both sides of every line."""
import pytest

SMS = 148


@pytest.fixture(scope="module")
def lib():
    from libtbvcoll_b200 import ops
    return ops.lib()


# 0 decode form, 1 / 2 tiles of 128 / 256 tokens
@pytest.mark.parametrize("M,rows,groups,K,epi,form", [
    (4096, 8 * 1024, 8, 7168, 0, 2), (4096, 4 * 4096, 4, 7168, 0, 2), (4096, 8 * 768, 8, 7168, 0, 2),       # long K, large groups, many rounds
    (4096, 8 * 512, 8, 7168, 0, 1), (4096, 16 * 500, 16, 7168, 0, 1),                                         # groups of few tiles
    (2048, 8 * 1024, 8, 7168, 0, 1),                                                                           # few rounds
    (4096, 8 * 1024, 8, 3584, 0, 1), (2048, 8 * 1024, 8, 3584, 0, 1),                                         # short K
    (14336, 8 * 1024, 8, 7168, 3, 1),                                                                          # an epilogue that computes
    (4096, 8 * 63, 8, 7168, 0, 0), (4096, 8 * 64, 8, 7168, 0, 1), (4104, 8 * 1024, 8, 7168, 0, 0), (4096, 513 * 800, 513, 7168, 0, 0)])
def test_row_grouped_products(lib, M, rows, groups, K, epi, form):
    assert lib.tbv_op_gemm_rows_form(M, rows, groups, K, epi, SMS) == form


@pytest.mark.parametrize("y,copy,many", [(4096, None, True), (4096, 8192, True), (4096, 8192 + 16, True), (4096, 8192 + 8, False), (4096 + 16, None, False), (4096 + 16, 8192, False)])
def test_results_and_copies_that_the_wide_stores_cannot_take(lib, y, copy, many):
    """fp32 results are stored 32 bytes at a time and their bf16 copy 16: a copy that is only 8-byte aligned (a slice of columns) goes to the form that stores 8."""
    assert (lib.tbv_op_gemm_ex_form(y, copy, 4096, 1024, 2048, 4096, 2, 1, SMS) > 0) == many
