"""Latent attention of portions on tcgen05 against float64, and bit for bit against the kernel on mma.sync: portions behind contexts, more rows and fewer than a tile, keys that end inside
a tile and inside a page, ranks of one to four blocks, pages nobody owns full of NaN, and a maximum that keeps growing."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def run(portions, heads, rank, rot, page, sinks, rising=False):
    from stride_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(heads + rank)
    randn = lambda *size: torch.randn(*size, generator=g, device="cuda")
    tokens, width = sum(n for _, n in portions), rank + rot
    counts = [-(-(p + n) // page) for p, n in portions]
    order = torch.randperm(sum(counts) + 3, generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.full((len(portions), max(counts)), -1, dtype=torch.int32)
    for i, c in enumerate(counts):
        table[i, :c], order = torch.tensor(order[:c], dtype=torch.int32), order[c:]
    latent, key_rot = (randn(sum(counts) + 3, 1, page, n).bfloat16() for n in (rank, rot))
    latent[order], key_rot[order] = float("nan"), float("nan")
    for i, (p, n) in enumerate(portions):           # and so is what lies behind the last key in its page
        if (p + n) % page:
            latent[table[i, counts[i] - 1], 0, (p + n) % page:], key_rot[table[i, counts[i] - 1], 0, (p + n) % page:] = float("nan"), float("nan")
    q = randn(tokens, heads, width)
    if rising:          # keys that point more and more the queries' way: the maximum grows by far more than 2^8 on the way
        q = q.abs()
        for i, (p, n) in enumerate(portions):
            for key in range(p + n):
                latent[table[i, key // page], 0, key % page] = latent[table[i, key // page], 0, key % page].abs() * (0.05 * key)
    q = q.bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    starts = [sum(n for _, n in portions[:i]) for i in range(len(portions))]
    sink = randn(heads) if sinks else None
    out = torch.full((tokens + 1, heads * rank), 7.0, device="cuda").bfloat16()
    scale = width ** -0.5
    took = ops.latent_attention_tc5(q.reshape(tokens, -1), out[:tokens], latent, key_rot, table.cuda(), i32(starts), i32([n for _, n in portions]),
                                    i32([p + n for p, n in portions]), len(portions), max(n for _, n in portions), heads, rank, rot, page, scale, sinks=sink)
    assert took and ops.tc_status() == 0 and bool((out[tokens] == 7.0).all())
    other, seq_of = torch.empty_like(out[:tokens]), i32(sum([[i] * n for i, (_, n) in enumerate(portions)], []))
    ops.latent_attention_tc(q.reshape(tokens, -1), other, None, latent, key_rot, table.cuda(), i32(starts), i32([n for _, n in portions]),
                            i32([p + n for p, n in portions]), seq_of, 0, len(portions), 0, tokens, max(2, max(n for _, n in portions)), heads, rank,
                            rot, page, scale, sinks=sink)
    assert torch.equal(out[:tokens], other)
    for i, (p, n) in enumerate(portions):
        at = torch.tensor([int(table[i, k // page]) * page + k % page for k in range(p + n)], device="cuda")
        c, r, mine = latent.view(-1, rank)[at].double(), key_rot.view(-1, rot)[at].double(), q[starts[i]:starts[i] + n].double()
        s = (torch.einsum("nhd,kd->nhk", mine[..., :rank], c) + torch.einsum("nhd,kd->nhk", mine[..., rank:], r)) * scale
        s = s.masked_fill(torch.arange(p + n, device="cuda")[None, None] > torch.arange(p, p + n, device="cuda")[:, None, None], float("-inf"))
        if sinks:
            s = torch.cat([s, sink.double()[None, :, None].expand(n, -1, 1)], -1)
        w = torch.softmax(s, -1)[..., :p + n]
        want, size = torch.einsum("nhk,kd->nhd", w, c), torch.einsum("nhk,kd->nhd", w, c.abs())
        # a probability (2^-8 of it), their sum (as rounded: as much) and the result (2^-8) are rounded to bfloat16; scores are float32 sums of
        # up to 576 terms, cut off every 16: 36 x 2^-23 of their terms' size, which with rising keys is some 2^9 (and 2^-9 the most it adds up to)
        got = out[starts[i]:starts[i] + n].view(n, heads, rank).double()
        assert bool(((got - want).abs() <= 2.0 ** -8 * (2.1 * size + want.abs()) + (2.0 ** -9 * size if rising else 0) + 1e-6).all()), \
            (i, float((got - want).abs().max()))


@pytest.mark.parametrize("portions,heads,rank,rot,page,sinks", [
    ([(0, 130)], 16, 512, 64, 16, True), ([(37, 61), (0, 1), (500, 9), (0, 200)], 5, 256, 16, 32, False), ([(100, 33)], 16, 128, 64, 8, True),
    ([(3, 70), (0, 3)], 3, 384, 48, 64, False), ([(63, 1), (64, 2), (0, 64), (0, 65)], 128, 512, 64, 16, False), ([(9, 7)], 1, 512, 32, 24, True)])
def test_against_float64(portions, heads, rank, rot, page, sinks):
    run(portions, heads, rank, rot, page, sinks)


def test_a_maximum_that_keeps_growing():
    run([(200, 100)], 16, 512, 64, 16, True, rising=True)


def test_sizes_that_are_left_to_the_other_kernel():
    from stride_b200.csrc import ops
    z, pages = torch.zeros(4, dtype=torch.int32, device="cuda"), lambda n: torch.zeros(2, 1, 16, n, dtype=torch.bfloat16, device="cuda")
    for rank, rot in ((80, 64), (512, 80), (256, 24)):
        q, out = torch.zeros(4, 2 * (rank + rot), dtype=torch.bfloat16, device="cuda"), torch.zeros(4, 2 * rank, dtype=torch.bfloat16, device="cuda")
        assert not ops.latent_attention_tc5(q, out, pages(rank), pages(rot), z.view(1, 4), z[:1], z[:1] + 4, z[:1] + 4, 1, 4, 2, rank, rot, 16, 1.0)
