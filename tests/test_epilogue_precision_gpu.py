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


# b = 2.17: the result passes through zero near z = -0.55, where errors of its parts stand out
@pytest.mark.parametrize("a, b", [(0.8, 40.0), (1.5, 0.9), (1.5, 2.17)])
@pytest.mark.parametrize("lo, hi", [(-9.0, -0.4), (-0.57, -0.53), (-0.6, 0.6), (-110.0, 3.0)])
@pytest.mark.parametrize("tokens", [7, 200, 2048])
def test_xielu(tokens, lo, hi, a, b, device):
    from ferrisinfer_b200.kernels import ops

    outputs = min(16384, max(512, 200000 // tokens // 64 * 64))
    x, w, _ = exact_inputs(tokens, outputs, lo, hi, device, 2)
    out = torch.empty(tokens, outputs, dtype=BF16, device=device)
    params = torch.tensor([a, b - 0.5], dtype=torch.float64).expm1().log().float().to(device)  # (what softplus takes to a and b - 1/2)
    ops.gemm_activation(x, w, out, "xielu", (a, b), params)
    z = x.double() @ w.double().t()
    a, b = float(torch.tensor(a).float()), float(torch.tensor(b).float())
    bend = torch.expm1(z) - z
    want = torch.where(z > 0, a * z * z + z / 2, b * bend + z / 2)
    # e^z - 1 to one unit of its last place; the difference, the product and the sum rounded to fp32; and the check's own rounding
    last = torch.ldexp(torch.ones_like(z), torch.frexp(torch.expm1(z))[1] - 24)
    error = torch.where(z > 0, 4 * 2.0 ** -24 * want.abs(), b * (last + 2.0 ** -24 * bend * (z < -2)) + 2 * 2.0 ** -24 * want.abs())
    assert_rounded(out, want, error)
    assert ops.kernel_status() == 0


@pytest.mark.parametrize("tokens", [7, 200, 2048])
def test_xielu_on_the_way_has_the_bits_of_its_own_kernel(tokens, device):
    """Where the product is a bf16 number, the kernel that other steps run behind it reads the same number."""
    from ferrisinfer_b200.kernels import ops

    z = torch.arange(2 ** 16, dtype=torch.int32).to(torch.int16).view(BF16)
    z = z[torch.isfinite(z) & (z.abs() >= 2.0 ** -14) & (z.abs() < 100)]
    z = torch.cat([z, torch.tensor([0.0, -0.0, float("inf"), -float("inf"), float("nan")], dtype=BF16)])
    w = torch.zeros(-(-len(z) // 64) * 64, 64, dtype=BF16)
    w[:len(z), 0] = z
    x = torch.zeros(tokens, 64, dtype=BF16, device=device)
    x[:, 0] = 1.0
    w, params = w.to(device), torch.tensor([30000.0, 30000.0], device=device)  # (softplus of 30,000 is 30,000 in fp32)
    out, plain = (torch.empty(tokens, w.shape[0], dtype=BF16, device=device) for _ in range(2))
    ops.gemm_activation(x, w, out, "xielu", (30000.0, 30000.5), params)
    ops.gemm(x, w, None, plain)
    ops.activation(plain, plain, "xielu", params)
    assert torch.equal(out.view(torch.int16), plain.view(torch.int16))
