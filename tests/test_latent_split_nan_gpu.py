"""A single token's keys in splits and in one run: what is no number in the last split's keys comes out of both, for every row of its request and
for no other's."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [2, 5, 40])
def test_no_number_in_the_last_split_is_not_lost(splits):
    from stride_b200.csrc import ops
    heads, rank, rot, page, contexts = 16, 128, 64, 16, [splits * 64, 70]
    g = torch.Generator(device="cuda").manual_seed(splits)
    pages = [-(-c // page) for c in contexts]
    table = torch.full((2, max(pages)), -1, dtype=torch.int32)
    table[0, :pages[0]], table[1, :pages[1]] = torch.arange(pages[0]), pages[0] + torch.arange(pages[1])
    latent, key_rot = (torch.randn(sum(pages), 1, page, n, generator=g, device="cuda").bfloat16() for n in (rank, rot))
    key_rot[pages[0] - 4:pages[0]] = float("nan")           # the scores of the first request's last 64 keys
    qa = torch.randn(2, heads * (rank + rot), generator=g, device="cuda").bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    outs = []
    for n in (1, splits):
        out = torch.zeros(2, heads * rank, device="cuda").bfloat16()
        partial = torch.zeros(2 * heads * n * (rank + 2), device="cuda") if n > 1 else None
        ops.latent_attention_tc(qa, out, partial, latent, key_rot, table.cuda(), i32([0, 1]), i32([1, 1]), i32(contexts), i32([0, 1]), 0, 2, 0, 2, 1, heads,
                                rank, rot, page, 0.07, splits=n, keys_per_split=64 if n > 1 else 0)
        outs.append(out.float())
    assert bool(outs[0][0].isnan().all()) and bool(outs[1][0].isnan().all())
    assert bool(outs[1][1].isfinite().all()) and float((outs[0][1] - outs[1][1]).abs().max()) < 2.0 ** -7 * float(outs[0][1].abs().max())
