"""Gate and up products of few tokens whose weights do not stand whole in shared memory, against 64 bits."""

import pytest
import torch

from test_kernels_gpu import rnd

pytestmark = pytest.mark.gpu

F32 = torch.float32


@pytest.mark.parametrize("T", [1, 8, 9, 16])
@pytest.mark.parametrize("I, K", [(18944, 3584), (8960, 1536), (9001, 1536), (11008, 4096), (6000, 1664)])
def test_gate_and_up_rows_in_passes(T, I, K, device):
    """Outputs eight at a time (an odd number of them at the end, K blocks that do not fill the last copy), from rows in bf16 and from
    rows to normalise; twice the same bits."""
    from ferrisinfer_b200.kernels import ops

    x, w = rnd((T, K), torch.bfloat16, device, 61), rnd((2 * I, K), torch.bfloat16, device, 62, 0.05)
    if not ops._skinny_takes(x, w, torch.empty(T, I, dtype=torch.bfloat16, device=device), 2):
        pytest.skip("left to the tcgen05 kernel")
    out, again = (torch.full((T, I + 1), float("nan"), dtype=torch.bfloat16, device=device) for _ in range(2))
    ops.gemm_skinny(x, w, None, out[:, :I], 3, up_row_offset=I)
    ops.gemm_skinny(x, w, None, again[:, :I], 3, up_row_offset=I)
    y = x.double() @ w.double().t()
    want = y[:, :I] * torch.sigmoid(y[:, :I]) * y[:, I:]
    # the result's rounding to 8 bits, and sums of K products in fp32
    limit = 2.0 ** -8 * want.abs() + K * 2.0 ** -22 * want.abs().max()
    assert ((out[:, :I].double() - want).abs() <= limit).all() and torch.equal(out[:, :I], again[:, :I]) and out[:, I].isnan().all()
    h, nw = rnd((T, K), F32, device, 63), 1 + rnd((K,), F32, device, 64, 0.1)
    lazy = ops.LazyRMSNorm(h, nw, 1e-6, torch.empty(T, K, dtype=torch.bfloat16, device=device))
    if not ops._skinny_takes(lazy, w, out[:, :I], 2):
        return
    rows = torch.empty(T, K, dtype=torch.bfloat16, device=device)
    ops.rmsnorm(h, nw, 1e-6, rows)
    ops.gemm_skinny(lazy, w, None, out[:, :I], 3, up_row_offset=I)
    y = rows.double() @ w.double().t()
    want = y[:, :I] * torch.sigmoid(y[:, :I]) * y[:, I:]
    assert (out[:, :I].double() - want).norm() <= 2.0 ** -8 * want.norm()
    assert ops.kernel_status() == 0
