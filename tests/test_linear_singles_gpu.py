"""Linear attention of steps of single tokens, where the states of many requests pass through rings of bulk copies: against the walk that
fewer requests take, and what it leaves alone."""

from types import SimpleNamespace

import pytest
import torch

from test_kernels_gpu import rnd

pytestmark = pytest.mark.gpu

F32, BF16 = torch.float32, torch.bfloat16


def context(slots, positions, device, lens=None):
    starts = [0]
    for n in lens or [1] * len(slots):
        starts.append(starts[-1] + n)
    to = lambda v: torch.tensor(v, dtype=torch.int32, device=device)
    return SimpleNamespace(max_q_len=1, num_seqs=len(slots), seq_q_start=to(starts), seq_state_slot=to(slots), positions=to(positions),
                           workspace=None)


# 1,536 tiles of 32 columns and one request more; tiles that do not divide among the CTAs; rotations whole, in part, of neighbours
@pytest.mark.parametrize("dtype, requests, heads, vdim, rotary, silu, write", [
    (BF16, 24, 16, 128, None, True, True), (BF16, 25, 16, 128, (128, False), False, True), (F32, 33, 12, 160, (64, True), False, True),
    (BF16, 70, 7, 128, (40, False), True, False), (BF16, 200, 3, 96, (128, True), False, True)])
def test_single_tokens_of_many_requests(dtype, requests, heads, vdim, rotary, silu, write, device):
    from ferrisinfer_b200.kernels import ops

    dim = 128
    assert requests * heads * vdim // 32 >= 1536
    q_size, v_size = heads * dim, heads * vdim
    qkv = rnd((requests, 2 * q_size + v_size + 16), dtype, device, 1)
    state = rnd((requests + 3, heads, vdim, dim), F32, device, 2)
    decay = 1.0 - torch.rand(heads, generator=torch.Generator().manual_seed(3)).to(device) * 0.2
    slots = torch.randperm(requests + 3, generator=torch.Generator().manual_seed(4))[:requests].tolist()
    positions = [37 * i % 4001 for i in range(requests)]
    table = None
    if rotary:
        n, neighbours = rotary
        table = ops.RotaryTable(10000.0 ** (-torch.arange(0, n, 2, device=device).float() / n), n, neighbours, 1.1)
    offsets = (0, q_size, 2 * q_size)
    out, want = torch.empty(requests, v_size, device=device), torch.empty(requests, v_size, device=device)
    mine, theirs = state.clone(), state.clone()
    ops.linear_attention(qkv, offsets, out, mine, decay, context(slots, positions, device), heads, dim, vdim, silu=silu, write_state=write,
                         rotary=table, k_scale=0.7 if rotary else 1.0)
    few = 1535 // (heads * vdim // 32)
    for i in range(0, requests, few):
        j = min(requests, i + few)
        ops.linear_attention(qkv[i:j], offsets, want[i:j], theirs, decay, context(slots[i:j], positions[i:j], device), heads, dim, vdim,
                             silu=silu, write_state=write, rotary=table, k_scale=0.7 if rotary else 1.0)
    # the same roundings in the same order
    assert torch.equal(mine, theirs) and torch.equal(mine, state) == (not write)
    assert torch.equal(out, want)
    assert ops.kernel_status() == 0


def test_requests_without_a_token_are_left_alone(device):
    from ferrisinfer_b200.kernels import ops

    heads, dim = 16, 128
    lens = [1, 0, 1, 1, 0, 0] * 9
    T, S = sum(lens), len(lens)
    qkv, state = rnd((T, 3 * heads * dim), BF16, device, 5), rnd((S, heads, dim, dim), F32, device, 6)
    out, before = torch.full((T, heads * dim), 7.0, device=device), state.clone()
    decay = torch.full((heads,), 0.9, device=device)
    ctx = context(list(range(S)), [0] * T, device, lens)
    ops.linear_attention(qkv, (0, heads * dim, 2 * heads * dim), out, state, decay, ctx, heads, dim, dim)
    q, k, v = (qkv[:, i * heads * dim:(i + 1) * heads * dim].double().view(T, heads, dim) for i in range(3))
    live = [i for i, n in enumerate(lens) if n]
    new = before[live].double() * decay.double()[0] + v.unsqueeze(-1) * k.unsqueeze(-2)
    assert torch.allclose(state[live].double(), new, rtol=1e-6, atol=1e-5)
    assert torch.allclose(out.double(), (new * q.unsqueeze(-2)).sum(-1).reshape(T, -1), rtol=1e-4, atol=1e-3)
    idle = [i for i, n in enumerate(lens) if not n]
    assert torch.equal(state[idle], before[idle])
