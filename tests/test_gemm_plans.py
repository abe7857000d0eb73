"""How products are divided among kernels; plans are made on the host."""

import pytest

from ferrisinfer_b200.kernels import ops


@pytest.mark.parametrize("N, K, rows_up_to", [(1152, 896, 32), (896, 896, 32), (9728, 896, 16), (896, 4864, 16), (2048, 1536, 16),
                                              (17920, 1536, 16), (1536, 8960, 16), (4608, 3584, 16), (3584, 3584, 16),
                                              (37888, 3584, 12), (3584, 18944, 3), (8, 4, 32), (40, 9220, 32)])
def test_32_bit_products_of_few_tokens_leave_long_rows_to_the_tiles(N, K, rows_up_to):
    """The kernel for few tokens reads the weights once for every so many tokens as fit; where it would read them too often
    the tiles take the product (the measured times stand beside the rule)."""
    taken = [ops.gemm_f32_plan(M, N, K) for M in range(1, 65)]
    assert all(t > 0 for t in taken[:rows_up_to]) and not any(taken[rows_up_to:])
    assert all(t <= 8 for t in taken) and taken[0] == 1


def test_swiglu_rides_along_where_the_rows_kernel_takes_both_products():
    for I, K in ((4864, 896), (8960, 1536), (18944, 3584), (40, 9220)):
        for M in (1, 4, 8, 12, 16):
            assert (ops.gemm_f32_plan(M, I, K, swiglu=True) > 0) == (ops.gemm_f32_plan(M, 2 * I, K) > 0), (I, K, M)
        assert ops.gemm_f32_plan(33, I, K, swiglu=True) == 0
