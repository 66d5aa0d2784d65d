"""The decayed memory with a bonus at head sizes around what four lanes a column hold (up to 64 rows; two columns a thread from 64 on), token by
token and in pieces, against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [32, 33, 40, 63, 64, 65])
@pytest.mark.parametrize("lengths", [(1, 1, 1), (130, 1, 70), (64, 65)])
def test_against_float64(D, lengths):
    from stride_b200.csrc import ops
    H, T, n = 2, sum(lengths), len(lengths)
    g = torch.Generator(device="cuda").manual_seed(D + T)
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    r, k, v = (rand(T, H * D) for _ in range(3))
    wlog, w0, bonus, state = rand(T, H * D), rand(H * D) - 3, rand(H * D), rand(n, H * D * D)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    starts = [sum(lengths[:i]) for i in range(n)]
    slots = list(range(n))[::-1]
    want, size = torch.zeros(T, H, D, dtype=torch.float64, device="cuda"), torch.zeros(T, H, D, dtype=torch.float64, device="cuda")
    ends = torch.empty(n, H, D, D, dtype=torch.float64, device="cuda")
    r64, k64, v64 = (x.double().view(T, H, D) for x in (r, k, v))
    keep, b64 = torch.exp(-torch.exp((wlog + w0).double())).view(T, H, D), bonus.double().view(H, D)
    for i in range(n):
        S = state[slots[i]].double().view(H, D, D)
        A = S.abs()
        for t in range(starts[i], starts[i] + lengths[i]):
            kv = k64[t][:, :, None] * v64[t][:, None, :]
            want[t] = ((S + b64[:, :, None] * kv) * r64[t][:, :, None]).sum(1)
            size[t] = ((A + (b64[:, :, None] * kv).abs()) * r64[t][:, :, None].abs()).sum(1)
            S, A = keep[t][:, :, None] * S + kv, keep[t][:, :, None] * A + kv.abs()
        ends[slots[i]] = S
    longest = max(lengths)
    for pieces in (False, True) if longest > 64 else (False,):
        o, s = torch.full((T, H * D), 7.0, device="cuda"), state.clone()
        scratch = torch.zeros(ops.bonus_scan_scratch_floats(n, longest, H, D), device="cuda") if pieces else None
        ops.bonus_scan(r, k, v, wlog, w0, bonus, o, s, i32(starts), i32(lengths), i32(slots), n, H, D, longest, scratch)
        # a term passes through at most T roundings of the memory, D of the sum, a few of its own and those of its decay's exponentials
        bound = (longest + D + 40) * 2.0 ** -24 * size
        assert bool(((o.double().view(T, H, D) - want).abs() <= bound).all()), pieces
        got = s.double().view(n, H, D, D)
        assert bool(((got - ends).abs() <= (longest + 40) * 2.0 ** -23 * ends.abs().amax((1, 2, 3), keepdim=True)).all()), pieces
