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
    assert ops._skinny_takes(x, w, torch.empty(T, I, dtype=torch.bfloat16, device=device), 2)
    # (beside 16 rows of 3,584 and 4,096 there is no room for a ring of copies)
    assert ops.gemm_skinny_plan(T, I, K, swiglu=True)["passes"] == (T <= 8 or K < 3584)
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
        assert T > 8  # (rows that are formed stand whole in shared memory)
        return
    assert ops.gemm_skinny_plan(T, I, K, swiglu=True, formed=True)["passes"] == (T <= 8 or K < 3584)
    rows = torch.empty(T, K, dtype=torch.bfloat16, device=device)
    ops.rmsnorm(h, nw, 1e-6, rows)
    ops.gemm_skinny(lazy, w, None, out[:, :I], 3, up_row_offset=I)
    y = rows.double() @ w.double().t()
    want = y[:, :I] * torch.sigmoid(y[:, :I]) * y[:, I:]
    assert (out[:, :I].double() - want).norm() <= 2.0 ** -8 * want.norm()
    assert ops.kernel_status() == 0


# in passes with rows from memory and rows to normalise, an output count that is no multiple of eight; whole slabs and rings
@pytest.mark.parametrize("T, I, K, formed, passes", [
    (1, 8960, 1536, False, True), (8, 9001, 1536, True, True), (16, 8960, 1536, False, True), (8, 18944, 3584, True, True), (16, 13824, 2560, False, True),
    (8, 18000, 1024, False, True), (8, 4864, 896, False, False), (8, 9472, 1408, True, False), (16, 18944, 3584, False, False)])
def test_products_of_few_tokens_are_added_up_in_one_order(T, I, K, formed, passes, device):
    """A warp adds up its runs of K blocks, then the eight warps' sums are added: the same outputs whether or not they go through in passes.
    Every output is the sum of 2^40 at one K block, 1 at another and -2^40 at a third, of which the 1 is kept or lost by the order."""
    from ferrisinfer_b200.kernels import ops

    plan = ops.gemm_skinny_plan(T, I, K, swiglu=True, formed=formed)
    assert plan["passes"] == passes
    g, blocks = torch.Generator().manual_seed(K + T), K // 64
    places = torch.stack([torch.randperm(blocks, generator=g)[:3] for _ in range(I)])
    first, last = places[:, :2].min(1).values, places[:, :2].max(1).values
    owner = lambda kb: (kb // plan["run"]) % 8
    # (inside a warp -2^40 + 1 may be cut off instead of rounded: no 1 where they would meet)
    one = torch.where((owner(places[:, 2]) == owner(last)) & (owner(first) != owner(last)), first, places[:, 2])
    terms = torch.zeros(I, blocks)
    at = torch.arange(I)
    terms[at, first], terms[at, last] = 2.0 ** 40, -(2.0 ** 40)
    terms[at, one] = torch.where(one == first, terms[at, one], torch.ones(I))
    sums = torch.zeros(I)  # in fp32, as the kernel adds: 2^40 + 1 is 2^40
    for warp in range(8):
        own = torch.zeros(I)
        for kb in range(blocks):
            if owner(kb) == warp:
                own = own + terms[:, kb]
        sums = sums + own
    assert 0.05 * I < (sums == 0).sum() < 0.95 * I and ((sums == 0) | (sums == 1)).all()
    w = torch.zeros(2 * I, blocks, 64, dtype=torch.bfloat16)
    w[:I, 0, 0], w[I:, :, 0] = 64.0, terms.to(torch.bfloat16)
    x = torch.zeros(T, blocks, 64)
    x[:, :, 0] = 1.0
    w, x = w.view(2 * I, K).to(device), x.view(T, K).to(device)
    rows = x.to(torch.bfloat16)
    if formed:  # an RMSNorm of rows whose mean square is 1/64, times 1/8
        rows = ops.LazyRMSNorm(x, torch.full((K,), 0.125, device=device), 0.0, torch.empty(T, K, dtype=torch.bfloat16, device=device))
    out = torch.empty(T, I, dtype=torch.bfloat16, device=device)
    ops.gemm_skinny(rows, w, None, out, 3, up_row_offset=I)
    assert torch.equal(out.float().cpu(), 64.0 * sums.expand(T, I))
    assert ops.kernel_status() == 0


@pytest.mark.parametrize("kind, limit", [("gelu_tanh", 0.0), ("clamped_swish", 1.5)])
@pytest.mark.parametrize("T, I", [(1, 8960), (8, 9001), (16, 8961)])
def test_other_gated_activations_in_passes(T, I, kind, limit, device):
    from ferrisinfer_b200.kernels import ops

    K = 1536
    x, w = rnd((T, K), torch.bfloat16, device, 65), rnd((2 * I, K), torch.bfloat16, device, 66, 0.05)
    assert ops.gemm_skinny_plan(T, I, K, swiglu=True)["passes"]
    out = torch.full((T, I + 1), float("nan"), dtype=torch.bfloat16, device=device)
    before = ops.launch_count()
    ops.gemm_gated(x, w, out[:, :I], kind, limit)
    assert ops.launch_count() - before == 1
    g, u = (x.double() @ w.double().t()).split(I, 1)
    if kind == "gelu_tanh":
        want = torch.nn.functional.gelu(g, approximate="tanh") * u
    else:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        want = g * torch.sigmoid(1.702 * g) * (u + 1)
    # as above
    assert ((out[:, :I].double() - want).abs() <= 2.0 ** -8 * want.abs() + K * 2.0 ** -22 * want.abs().max()).all() and out[:, I].isnan().all()
    assert ops.kernel_status() == 0
