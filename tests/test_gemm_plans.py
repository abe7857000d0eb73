"""How products are divided among kernels; plans are made on the host."""

import os
import subprocess
import sys

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


@pytest.mark.parametrize("T, I, K, blocks", [
    (8, 18944, 3584, 15), (16, 18944, 3584, 0), (8, 8960, 1536, 13), (16, 8960, 1536, 13), (1, 9001, 1536, 13), (8, 11008, 4096, 13),
    (9, 11008, 4096, 0), (8, 5632, 2048, 11), (16, 13824, 2560, 11), (8, 4864, 896, 0), (8, 9472, 1408, 0), (8, 9536, 1408, 11), (8, 18000, 896, 0),
    (8, 18000, 1024, 9)])
def test_gate_and_up_products_of_few_tokens_that_go_through_in_passes(T, I, K, blocks):
    """Where the weights of a CTA do not stand whole in shared memory and enough of them fit beside the step's rows (the measured times stand
    beside the rule); 0: the other kernel's."""
    plan = ops.gemm_skinny_plan(T, I, K, swiglu=True)
    assert plan["passes"] == (blocks > 0) and (not blocks or plan["blocks"] == blocks)
    assert not ops.gemm_skinny_plan(T, I, K)["passes"]


@pytest.mark.parametrize("kb", [60, 128, 160, 200, 219])
def test_passes_keep_to_the_shared_memory_that_was_asked_for(kb):
    code = ("from ferrisinfer_b200.kernels import ops\n"
            "for T, I, K in ((1, 8960, 1536), (16, 8960, 1536), (8, 18944, 3584), (8, 18000, 1024), (8, 4864, 896)):\n"
            "    if not ops._lib().ferris_gemm_skinny_takes(T, I, K, 2, 1):\n"
            "        continue\n"
            "    plan = ops.gemm_skinny_plan(T, I, K, swiglu=True)\n"
            f"    assert not plan['passes'] or plan['smem'] <= {kb} * 1024 + 1024, (T, I, K, plan)\n")
    subprocess.run([sys.executable, "-c", code], check=True, env={**os.environ, "FERRIS_SKINNY_SMEM_KB": str(kb)},
                   cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
