"""The matrix LSTM token by token with more requests than run side by side: every CTA of a head starts from what the head held before the
step, however late it comes. Outputs and states against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 3])
@pytest.mark.parametrize("H,D,DV,requests", [(16, 128, 128, 3), (16, 128, 128, 64), (8, 64, 96, 100), (4, 256, 256, 40), (16, 16, 16, 64)])
def test_every_column_starts_from_the_state_before(H, D, DV, requests, tokens):
    from stride_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(H + D + requests)
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    T, cap = requests * tokens, 15.0
    proj, gates, b_i, b_f = rand(T, 2 * H * D + H * DV), 2 * rand(T, 2 * H), rand(H), rand(H)
    state = rand(requests, H * D * DV + H * D + H)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    order = torch.randperm(requests, generator=torch.Generator().manual_seed(1)).tolist()
    o, got = torch.zeros(T, H * DV, device="cuda"), state.clone()
    tickets = torch.zeros(requests * H, dtype=torch.int32, device="cuda")
    ops.mlstm_scan(proj, 0, H * D, 2 * H * D, gates, b_i, b_f, cap, D ** -0.5, o, got, i32([tokens * r for r in range(requests)]), i32([tokens] * requests),
                   i32(order), requests, H, D, DV, tickets=tickets)
    assert not bool(tickets.any())
    rows = state[order].double()
    S, n, m = rows[:, :H * D * DV].view(-1, H, D, DV).clone(), rows[:, H * D * DV:-H].view(-1, H, D).clone(), rows[:, -H:].clone()
    x = proj.double().view(requests, tokens, -1)
    q, k = (x[..., i * H * D:(i + 1) * H * D].view(requests, tokens, H, D) for i in (0, 1))
    v, z = x[..., 2 * H * D:].view(requests, tokens, H, DV), gates.double().view(requests, tokens, 2 * H)
    for t in range(tokens):
        li, lf = cap * torch.tanh((z[:, t, :H] + b_i) / cap), torch.nn.functional.logsigmoid(cap * torch.tanh((z[:, t, H:] + b_f) / cap))
        new = torch.maximum(lf + m, li)
        keep, take = torch.exp(lf + m - new), torch.exp(li - new)
        S = keep[..., None, None] * S + take[..., None, None] * k[:, t, :, :, None] * v[:, t, :, None, :]
        n, m = keep[..., None] * n + take[..., None] * k[:, t], new
        query = q[:, t] * D ** -0.5
        num, dot = (S * query[..., None]).sum(2), (n * query).sum(2)
        den = torch.maximum(dot.abs(), torch.exp(-m)) + 1e-6
        # sums of D terms, exponentials of numbers up to 30 (32 x 2^-24 of them) and the quick quotient
        few = (D + 60 + 30 * t) * 2.0 ** -24
        size_num, size_dot = (S.abs() * query.abs()[..., None]).sum(2), (n.abs() * query.abs()).sum(2)
        bound = few * (size_num / den[..., None] + num.abs() * ((size_dot + den) / den ** 2)[..., None])
        mine = o.view(requests, tokens, H, DV)[:, t].double()
        assert bool(((mine - num / den[..., None]).abs() <= bound).all()), t
    back = got[order].double()
    few = (60 + 30 * tokens) * 2.0 ** -24
    for mine, want in ((back[:, :H * D * DV].view_as(S), S), (back[:, H * D * DV:-H].view_as(n), n), (back[:, -H:], m)):
        scale = want.abs().amax(tuple(range(2, want.dim())), keepdim=True) if want.dim() > 2 else want.abs() + 1
        assert bool(((mine - want).abs() <= few * scale).all())
