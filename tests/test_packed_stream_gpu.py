"""The stream beside its second input, and a vector on every row, four numbers a thread and one: the same bits from buffers on their boundaries
and off them, at widths that are whole packs and that are not."""

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
    x, y, vector = (torch.randn(*size, generator=g, device="cuda") for size in ((tokens, hidden), (tokens, hidden), (hidden,)))
    y = y.to(dtype)
    seq_of = torch.zeros(tokens, dtype=torch.int32, device="cuda")
    seq_of[tokens // 2] = -1
    for place in (torch.clone, shifted):
        out = place(torch.zeros(tokens, 2 * hidden, device="cuda", dtype=dtype))
        ops.stream_concat(place(x), place(y), out)
        assert torch.equal(out, torch.cat([x.to(dtype), y], 1))
        for seqs in (None, seq_of):
            row = place(x)
            ops.add_row_vector(row, place(vector), seqs)
            want = x + vector
            if seqs is not None:
                want[tokens // 2] = x[tokens // 2]
            assert torch.equal(row, want)
