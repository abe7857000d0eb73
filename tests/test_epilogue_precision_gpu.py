"""Activations in the epilogues of tensor-core products: what is rounded to bf16 is the fp32 value of the full functions.

The products themselves are exact here (one bf16 number times another), so a result is the rounding to bf16 of a number that lies within
the fp32 functions' error of the 64-bit one; a larger error shows where the 64-bit value lies close to the middle between two bf16 numbers."""

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = torch.bfloat16


def exact_inputs(tokens, outputs, lo, hi, device, seed):
    """x [tokens, 64] and w [outputs, 64] of which x w^T has one product each, spread over lo .. hi; and a column for another product."""
    g = torch.Generator().manual_seed(seed)
    x, w = torch.zeros(tokens, 64), torch.zeros(outputs, 64)
    x[:, 0] = 0.5 + torch.rand(tokens, generator=g) / 2
    w[:, 0] = lo + (hi - lo) * torch.rand(outputs, generator=g)
    return x.to(device, BF16), w.to(device, BF16), g


def assert_rounded(out, want, error):
    """out [bf16] is the rounding of a number within `error` of the 64-bit numbers `want`."""
    low, high = (want - error).float().to(BF16), (want + error).float().to(BF16)  # (fp32 first: a rounding that `error` has to cover)
    assert ((out >= low) & (out <= high)).all(), int(((out < low) | (out > high)).sum())


# few tokens (a product too tall for the kernel of few tokens), short steps and long ones (with and without CTA pairs)
@pytest.mark.parametrize("tokens", [7, 24, 64, 200, 512, 2048])
def test_swiglu(tokens, device):
    from ferrisinfer_b200.kernels import ops

    outputs = max(512, 200000 // tokens // 64 * 64)
    x, gate, g = exact_inputs(tokens, outputs, -85.0, 10.0, device, 1)
    up = torch.zeros(outputs, 64)
    up[:, 1] = 1 + 3 * torch.rand(outputs, generator=g)
    x[:, 1] = (1 + torch.rand(tokens, generator=g)).to(device, BF16)
    w = torch.cat([gate, up.to(device, BF16)])
    out = torch.empty(tokens, outputs, dtype=BF16, device=device)
    ops.gemm_swiglu(x, w, out)
    y = x.double() @ w.double().t()
    want = y[:, :outputs] * torch.sigmoid(y[:, :outputs]) * y[:, outputs:]
    # the exponential to two units of 2^-23, four roundings to fp32 and the one of the check
    assert_rounded(out, want, 9 * 2.0 ** -24 * want.abs())
    assert ops.kernel_status() == 0


@pytest.mark.parametrize("tokens", [24, 200, 2048])
def test_swiglu_of_the_largest_numbers(tokens, device):
    from ferrisinfer_b200.kernels import ops

    inf, nan = float("inf"), float("nan")
    gates = [-inf, -3e38, -200.0, -104.0, -89.0, -88.5, -88.0, -87.0, 0.0, -0.0, 88.0, 89.0, 200.0, 3e38, inf, nan]
    ups = [1.0, -2.0, 0.0, 3e38, inf, nan]
    n = len(gates) * len(ups)
    w = torch.zeros(2 * n, 64)
    w[:n, 0] = torch.tensor(gates).repeat_interleave(len(ups))
    w[n:, 0] = torch.tensor(ups).repeat(len(gates))
    w, x = w.to(device, BF16), torch.zeros(tokens, 64, device=device, dtype=BF16)
    x[:, 0] = 1.0
    out = torch.empty(tokens, n, dtype=BF16, device=device)
    ops.gemm_swiglu(x, w, out)
    g, u = w[:n, 0].float(), w[n:, 0].float()
    want = (u * (g * (1.0 / (1.0 + torch.exp(-g))))).to(BF16).expand(tokens, n)
    # (2^-126 and less: of the last bit of a number that bf16 holds with few bits)
    assert torch.allclose(out.float(), want.float(), rtol=2.0 ** -7, atol=2.0 ** -132, equal_nan=True)
    assert ops.kernel_status() == 0
