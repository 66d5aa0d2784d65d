"""What the gated delta rule's scan reads, against float64: portions that begin inside a warp's run of tokens, portions shorter than the
convolution, padded rows, one token a request, heads of odd sizes, both element types."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("portions,pad,G,H,D,DV", [([1, 1, 1], 1, 2, 4, 128, 128), ([5, 2, 1, 9, 30], 0, 3, 3, 40, 72), ([700, 1, 3, 333, 1], 2, 4, 8, 128, 96),
                                                 ([257], 0, 1, 30, 8, 128)])
def test_against_float64(portions, pad, G, H, D, DV, dtype):
    from stride_b200.csrc import ops
    taps, eps, C = 4, 1e-6, 2 * G * D + H * DV
    g = torch.Generator().manual_seed(D)
    randn = lambda *size: torch.randn(*size, generator=g)
    tokens, seqs = sum(portions) + pad, len(portions)
    proj, conv_w, low = randn(tokens, C + H + 3).to(dtype), randn(C, taps), randn(tokens, H * D + 2)
    a_log, dt_bias, state = randn(H) * 0.5, randn(H * D), randn(seqs + 2, 10 + (taps - 1) * C)
    starts = [sum(portions[:i]) for i in range(seqs)]
    seq_of = torch.tensor(sum([[i] * n for i, n in enumerate(portions)], []) + [-1] * pad, dtype=torch.int32)
    slots = torch.tensor([(i * 2 + 1) % (seqs + 2) for i in range(seqs)], dtype=torch.int32)
    dev = lambda t: t.cuda()
    qk, v, beta, decay = (torch.full((tokens, n), 7.0, device="cuda") for n in (2 * G * D, H * DV, H, H * D))
    ops.delta_prepare(dev(proj), dev(conv_w), dev(low), dev(a_log), dev(dt_bias), dev(state), 10, dev(seq_of), dev(torch.tensor(starts, dtype=torch.int32)),
                      dev(slots), qk, v, beta, decay, G, H, D, DV, taps, eps)
    x, want_c = proj.double(), torch.zeros(tokens, C, dtype=torch.float64)
    for i, n in enumerate(portions):
        tail = state[int(slots[i]), 10:].double().view(taps - 1, C)
        rows = torch.cat([tail, x[starts[i]:starts[i] + n, :C]])
        y = sum(rows[j:j + n] * conv_w[:, j].double() for j in range(taps))
        want_c[starts[i]:starts[i] + n] = y * torch.sigmoid(y)
    unit = want_c[:, :2 * G * D].view(tokens, 2, G, D)
    unit = unit / torch.sqrt((unit * unit).sum(-1, keepdim=True) + eps)
    unit[:, 0] *= D ** -0.5
    live = (seq_of >= 0).double()[:, None]
    want_decay = torch.expm1(-torch.exp(a_log.double()).repeat_interleave(D) * torch.nn.functional.softplus(low[:, :H * D].double() + dt_bias.double()))
    # float32 sums of four products, SiLU and the norm by a few units in the last place each
    for got, want in ((qk, unit.reshape(tokens, -1)), (v, want_c[:, 2 * G * D:]), (beta, torch.sigmoid(x[:, C:C + H])), (decay, want_decay)):
        want = want * live
        assert float((got.double().cpu() - want).abs().max()) < 4e-6 * max(1.0, float(want.abs().max()))
