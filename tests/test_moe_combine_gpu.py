"""The sum of a token's expert rows, four columns a thread and one: every count of experts at the edges of the two, rows left out, with and
without weights, shared expert and gate, against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("top,hidden,tokens", [(1, 4, 3), (3, 516, 5), (4, 2048, 9), (5, 520, 2), (8, 132, 4), (9, 256, 3), (4, 50, 3)])
def test_against_float64(top, hidden, tokens, dtype):
    from stride_b200.csrc import ops
    g = torch.Generator().manual_seed(top * hidden)
    randn = lambda *size: torch.randn(*size, generator=g)
    y, weights, shared, gates = randn(tokens * top + 2, hidden), randn(tokens, top), randn(tokens, hidden).to(dtype), randn(tokens, 3)
    row_of = torch.randperm(tokens * top + 2, generator=g)[:tokens * top].view(tokens, top).int()
    row_of[0, top - 1] = -1
    for use_rows, use_weights, use_shared, use_gate in ((1, 1, 1, 1), (1, 0, 1, 0), (0, 1, 0, 0), (1, 1, 0, 0), (0, 0, 1, 1)):
        rows = row_of.long() if use_rows else torch.arange(tokens * top).view(tokens, top)
        w = (weights.double() if use_weights else torch.ones(tokens, top, dtype=torch.float64)) * (rows >= 0)
        own = torch.sigmoid(gates[:, 1:2].double()) if use_gate else 1.0
        want = (y.double()[rows.clamp(min=0)] * w[..., None]).sum(1) + (own * shared.double() if use_shared else 0.0)
        out = torch.full((tokens + 1, hidden), 7.0, device="cuda", dtype=dtype)
        yd = y.cuda() if use_rows else y[:tokens * top].contiguous().cuda()
        ops.moe_combine(yd, row_of.cuda() if use_rows else None, weights.cuda() if use_weights else None, shared.cuda() if use_shared else None, out[:tokens],
                        shared_gate=gates.cuda()[:, 1] if use_gate else None)
        # top + 1 rounded float32 sums, then the result's element type
        size = (y.double()[rows.clamp(min=0)].abs() * w.abs()[..., None]).sum(1) + shared.double().abs()
        bound = (top + 3) * 2.0 ** -24 * size + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0.0) + 1e-7
        assert bool(((out[:tokens].cpu().double() - want).abs() <= bound).all()) and bool((out[tokens] == 7.0).all())
