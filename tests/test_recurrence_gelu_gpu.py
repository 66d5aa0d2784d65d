"""The gelu branch behind the linear recurrence, over its whole range and at its ends, against float64; token by token in 32 bits and in pieces."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def values():
    mid = torch.linspace(-14.0, 14.0, 4001)
    ends = torch.tensor([0.0, -0.0, 1e-30, -1e-30, 3e-39, -3e-39, -20.0, -1e3, -1e15, -3e38, 20.0, 1e3, 1e15, 3e38, math.inf, -math.inf, math.nan])
    return torch.cat([mid, ends])


def gelu(z):
    z = z.double()
    inner = math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)
    return z * torch.sigmoid(2.0 * inner), inner.abs()


@pytest.mark.parametrize("pieces", [False, True])
def test_gelu_over_its_range(pieces):
    from stride_b200.csrc import ops
    dtype, tokens, taps = (torch.bfloat16, 300, 4) if pieces else (torch.float32, 3, 4)
    z = values().to(dtype)
    width = z.numel()
    xy = torch.zeros(tokens, 2 * width, dtype=dtype)
    xy[:, :width] = z
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    zeros = lambda *shape: torch.zeros(*shape, device="cuda")
    state = zeros(1, taps, width)
    state[0, taps - 1] = 1.0                    # a - 1 = 0 and no input: S stays 1 and the output is the branch itself
    out = torch.empty(tokens, width, dtype=dtype, device="cuda")
    a, gx, b = zeros(tokens, width), zeros(tokens, width), zeros(width)
    where = (state, i32([0]), i32([tokens]), i32([0]), out)
    if pieces:
        ops.rglru_scan_pieces(a, gx, xy.cuda(), width, 0, b, b, *where, zeros((tokens // 64 + 2) * 2 * width), 1, tokens, taps)
    else:
        ops.rglru_scan(a, gx, xy.cuda(), width, 0, b, b, *where, 1, taps)
    want, inner = gelu(z)
    assert torch.equal(out, out[:1].expand_as(out)) or bool(out.isnan().any())
    got = out[-1].cpu().double()
    # both forms of the formula: minus infinity times nothing
    assert bool(got[z == -math.inf].isnan().all()) and bool(got[z.isnan()].isnan().all()) and bool((got[z == math.inf] == math.inf).all())
    ok = z.isfinite()
    # 2 y has six roundings, which the exponential takes times its argument (up to 89, beyond which it is
    # infinite); exponential, sum, quotient and, in 16 bits, the result: a few places more
    argument = (2 * inner).clamp(max=89.0)
    bound = want.abs() * (6 * argument * 2.0 ** -24 + 2.0 ** -21 + (2.0 ** -8 if pieces else 0.0)) + 2.0 ** -124      # (below, the exponential is infinite and the result 0)
    assert bool(((got - want).abs()[ok] <= bound[ok]).all())
