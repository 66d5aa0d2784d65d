"""A chunk's tokens and a number that is none: it comes out of the token that brings it and of those after it, in its head (and, in a value, in its
column), and of none before, as token by token. Constant decays, channel decays, the matrix LSTM and the state space."""

import pytest
import torch

pytestmark = pytest.mark.gpu

H, D, DV, LENGTHS = 3, 64, 128, (150, 100)


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def both(ops, rule, proj, logit, gates, state):
    """Outputs and states token by token and chunk by chunk."""
    starts, lens, slots, n, longest = i32([0, LENGTHS[0]]), i32(LENGTHS), i32([1, 0]), len(LENGTHS), max(LENGTHS)
    places, outs = (0, H * D, 2 * H * D), []
    for chunks in (False, True):
        o, s = torch.zeros(sum(LENGTHS), H * DV, device="cuda"), state.clone()
        tail = (o, s, starts, lens, slots, n, H, D, DV)
        if rule == "lstm":
            args = (proj, *places, gates, torch.zeros(H, device="cuda"), torch.ones(H, device="cuda"), 15.0, D ** -0.5, *tail)
            if chunks:
                ops.mlstm_chunks(*args, longest, torch.zeros(ops.mlstm_chunks_scratch_floats(n, longest, H, D, DV), device="cuda"))
            else:
                ops.mlstm_scan(*args)
        else:
            keep = torch.tensor([0.5, 0.9, 0.99], dtype=torch.float64, device="cuda")
            fading = rule == "constant"
            if chunks:
                form = (keep[:, None] ** torch.arange(65, device="cuda")).float() if fading else None
            else:
                form = (keep - 1).float() if fading else None
            bias = None if fading else torch.zeros(H * D, device="cuda")
            args = (proj, *places, None if fading else logit.clone(), bias, form, 1.0 if fading else D ** -0.5, 1.0 if fading else 1 / 16, *tail)
            if chunks:
                ops.decay_chunks(*args, longest, torch.zeros(ops.decay_chunks_scratch_floats(n, longest, H, D, DV), device="cuda"))
            else:
                ops.decay_scan(*args)
        outs.append((o, s))
    return outs


def inputs(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    T = sum(LENGTHS)
    return r(T, 2 * H * D + H * DV).bfloat16(), r(T, H * D) + 2, r(T, 2 * H), 0.1 * r(2, H * D * DV + H * D + H)


@pytest.mark.parametrize("what", ["value", "key", "infinite value"])
@pytest.mark.parametrize("rule", ["constant", "channel", "lstm"])
def test_no_number_stays_out_of_the_tokens_before_it(rule, what):
    from stride_b200.csrc import ops
    proj, logit, gates, state = inputs(1)
    # the first, a middle and the last token of eight; a chunk's last and the next one's first; the second request's broken chunk
    for t, head in ((0, 0), (3, 1), (61, 2), (LENGTHS[0] - 1, 0), (LENGTHS[0] + 63, 1), (LENGTHS[0] + 69, 2)):
        place = H * D + head * D + 5 if what == "key" else 2 * H * D + head * DV + 9
        proj[t, place] = float("inf") if what == "infinite value" else float("nan")
    (o, s), (oc, sc) = both(ops, rule, proj, logit, gates, state)
    assert torch.equal(o.isfinite(), oc.isfinite()) and torch.equal(s.isfinite(), sc.isfinite())
    ok = o.isfinite()
    assert bool(ok[LENGTHS[0] + 62].all()) and not bool(ok[LENGTHS[0] + 63].all())
    # sums of up to 150 terms of about 1 in another order, and the decays as products or as exponentials of sums: 2^-24 a step
    assert float((o[ok] - oc[ok]).abs().max()) < 300 * 2.0 ** -24 * float(o[ok].abs().max()) * D ** 0.5


def test_a_decay_that_is_no_number_leaves_the_strong_decays_before_it():
    from stride_b200.csrc import ops
    proj, logit, gates, state = inputs(2)
    logit[:40] = -160.0         # e^-10 a token: their products fall below what float32 can turn round
    logit[45, :D] = float("nan")        # every channel of the first head: none is left to tell of the strong ones
    (o, _), (oc, _) = both(ops, "channel", proj, logit, gates, state)
    assert torch.equal(o.isnan(), oc.isnan()) and bool(oc[:45].isfinite().all()) and bool(oc[45, :DV].isnan().all())
    ok = o.isfinite()
    assert float((o[ok] - oc[ok]).abs().max()) < 300 * 2.0 ** -24 * float(o[ok].abs().max()) * D ** 0.5


@pytest.mark.parametrize("what", ["value", "key", "infinite value"])
@pytest.mark.parametrize("P,N", [(64, 64), (72, 128)])
def test_state_space_chunks(P, N, what):
    from stride_b200.csrc import ops
    G, T = 1, sum(LENGTHS)
    g = torch.Generator(device="cuda").manual_seed(P)
    r = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    channels = H * P + 2 * G * N
    shape = ops.SsmShape(H, G, N, P, 4, r(H), r(H), r(H), r(4, channels), r(channels))
    u, raw, proj, state = r(T, channels).bfloat16(), r(T, H), r(T, channels).bfloat16(), 0.1 * r(2, shape.state_floats())
    # the first, a middle and the last token of sixteen; a chunk's last and the next one's first; the second request's broken chunk
    for t, head in ((0, 0), (5, 1), (127, 2), (LENGTHS[0] - 1, 0), (LENGTHS[0] + 63, 1), (LENGTHS[0] + 69, 2)):
        u[t, H * P + 3 if what == "key" else head * P + 9] = float("inf") if what == "infinite value" else float("nan")
    starts, lens, slots, positions = i32([0, LENGTHS[0]]), i32(LENGTHS), i32([1, 0]), i32([t for n in LENGTHS for t in range(n)])
    y, yc = (torch.zeros(T, H * P, device="cuda") for _ in range(2))
    s, sc = state.clone(), state.clone()
    ops.ssm_scan(shape, u, raw, 0, y, s, starts, lens, slots, 2)
    scratch = torch.zeros(ops.ssm_chunks_scratch_floats(shape, 2, max(LENGTHS)), device="cuda")
    ops.ssm_chunks(shape, u, raw, 0, yc, sc, proj, 0, starts, lens, positions, slots, 2, max(LENGTHS), scratch)
    memory = H * N * P
    assert torch.equal(y.isfinite(), yc.isfinite()) and torch.equal(s[:, :memory].isfinite(), sc[:, :memory].isfinite())
    ok = y.isfinite()
    assert bool(ok[LENGTHS[0] + 62].all()) and not bool(ok[LENGTHS[0] + 63].all())
    # operands of two bfloat16 parts (2^-16 of a term, of which a sum has N and 64)
    assert float((y[ok] - yc[ok]).abs().max()) < 2.0 ** -13 * float(y[ok].abs().max())
