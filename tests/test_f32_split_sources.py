"""The split products take tensor memory before they let dependents in, as the kernels of test_kernel_sources.py do."""

from test_kernel_sources import kernels_with


def test_the_split_products_take_tensor_memory_before_dependents_are_let_in():
    (_, kernel, body), = kernels_with("take_tensor_memory")
    assert kernel == "gemm_f32_split_kernel"
    assert body.index("take_tensor_memory") < body.index("pdl_launch_dependents()")
    assert body.count("pdl_launch_dependents()") == 1
