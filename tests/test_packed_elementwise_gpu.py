"""Dynamic Tanh with its sum, the scaled sum and the cast, four elements a thread and one: the same bits from buffers on their boundaries and
off them, at widths that are whole packs and that are not, with and without a delta and chosen rows."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def shifted(t):
    """The same values one element off a 16-byte boundary."""
    room = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    room.copy_(t)
    return room


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,hidden", [(1, 4), (3, 1020), (5, 1028), (70, 2048), (2, 50)])
def test_packs_and_single_elements_agree(tokens, hidden, dtype):
    from stride_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(hidden)
    randn = lambda *size: torch.randn(*size, generator=g, device="cuda")
    res, delta, w, b = randn(tokens, hidden), randn(tokens, hidden).to(dtype), randn(hidden), randn(hidden)
    rows = torch.randint(0, tokens, (tokens + 2,), generator=g, device="cuda", dtype=torch.int32)
    for d, pick in ((delta, None), (None, None), (delta, rows)):
        outs = []
        for place in (torch.clone, shifted):
            r, out = place(res), place(torch.zeros(tokens if pick is None else tokens + 2, hidden, device="cuda", dtype=dtype))
            ops.add_dyt(r, d if d is None else place(d), 0.5, w, b, 0.7, out, rows=pick)
            outs.append((r.clone(), out.clone()))
        assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
        x = res.double() + (0.5 * d.double() if d is not None else 0.0)
        want = torch.tanh(0.7 * (x if pick is None else x[pick.long()])) * w.double() + b.double()
        assert float((outs[0][1].double() - want).abs().max()) < (2.0 ** -7 if dtype == torch.bfloat16 else 2e-6) * max(1.0, float(want.abs().max()))
    sums = [place(res) for place in (torch.clone, shifted)]
    for s, place in zip(sums, (torch.clone, shifted)):
        ops.add_scaled(s, place(delta), 0.25)
    assert torch.equal(*sums) and float((sums[0].double() - res.double() - 0.25 * delta.double()).abs().max()) < 1e-6
    casts = [torch.full((tokens, hidden), 7.0, device="cuda", dtype=dtype) for _ in range(2)]
    for c, place in zip(casts, (torch.clone, shifted)):
        ops.cast_rows(place(res), c)
    assert torch.equal(*casts) and torch.equal(casts[0], res.to(dtype))
