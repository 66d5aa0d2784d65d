"""The Netusun decoder in the engine against the plain float64 implementation (``plain_netusun``): each mechanism alone (as a
kernel and in a model of nothing else), the stream after every layer run, whole prompts against token-by-token decoding,
portions down to two tokens, batches of unequal requests on pages and state slots that are used again, keys just inside and
just outside a window in prompts and among decoded tokens, a far past that only sharp latent attention or a slow-forgetting
memory still shows, the first tokens, long decoding, sizes unlike one another, and greedy generation through the engine's
scheduler."""

import copy
import math

import pytest
import torch

import netusun_cases as cases
import plain_netusun as plain
import trace_modes as modes
from helpers import compare_logits, seeded_tokens, write_model_dir

pytestmark = pytest.mark.gpu
STORED = {"float32": torch.float32, "bfloat16": torch.bfloat16}


@pytest.fixture(scope="module")
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def close(got, want, tol):
    got, want = got.double().cpu(), want.double().cpu()
    scale = float(want.abs().max())
    err = float((got - want).abs().max())
    assert err <= tol * scale, f"max abs error {err:.3e} against scale {scale:.3e}"


BF16_BOUND = (0.998, 0.06)          # cosine floor and largest error of a row relative to its spread
BF16_BOUND_DEEP = (0.99, 0.15)      # eight runs with sixteen experts: measured, the error grows from 0.4 % of the stream after
#                                     the first run to 2.6 % after the last, and a router's close call moves single rows by 10 %


def compare_rows(got, want, dtype, bound=BF16_BOUND):
    """float32: the helpers' bound (cosine and largest difference). bfloat16: what the rounding of activations leaves of a
    row, a few per cent of its spread for these small random models; a wrong key, window or expert changes a row outright,
    and the float32 runs of the same cuttings hold the tight bound."""
    if dtype == "float32":
        return compare_logits(got, want, dtype)
    a, b = got.double().reshape(-1), want.double().reshape(-1)
    if not torch.isfinite(a).all():
        return False, "non-finite logits"
    cos = float(torch.nn.functional.cosine_similarity(a, b, dim=0))
    rel = float((a - b).norm() / (b - b.mean()).norm())
    return cos >= bound[0] and rel <= bound[1], f"cosine {cos:.6f}, error {rel:.3f} of the row's spread"


def rounded(state, dtype):
    return {k: v.to(STORED[dtype]) for k, v in state.items()}


def replay(folder, dtype, steps, want, page, slots, label, min_ok=1.0, bound=BF16_BOUND):
    """Runs the steps through a fresh session and compares every wanted row; pages and state slots start as NaN."""
    from stride_b200.engine.trace import TraceSession
    session = TraceSession(folder, dtype, max_tokens=modes.peak_tokens(steps), block_size=page, max_requests=slots)
    for t in list(session.device_cache.pages) + list(session.device_cache.states.values()):
        t.fill_(float("nan"))
    rows = modes.expected_rows(steps)
    bad, total, first = 0, 0, None
    for s in steps:
        out = session.run_step(s)
        for r, (rid, pos) in enumerate(rows[s["step"]]):
            ok, msg = compare_rows(out[r:r + 1], want[rid][pos:pos + 1], dtype, bound)
            total += 1
            if not ok:
                bad += 1
                first = first or f"{label}: step {s['step']}, request {rid!r}, position {pos}: {msg}"
    assert total and bad <= (1.0 - min_ok) * total, f"{bad} of {total} rows differ; first: {first}"
    stats = session.cache.stats()
    assert stats["live"] == 0 and session.cache.free_slots == session.cache.slot_capacity
    return session


def model_case(tmp_models, name, cfg, dtype, seed, lengths, **state_options):
    state = cases.seeded_state(cfg, seed, **state_options)
    folder = write_model_dir(str(tmp_models / f"netusun_{name}_{dtype}_{seed}"), cfg, state, STORED[dtype])
    state = {k: v.double() for k, v in rounded(state, dtype).items()}
    requests = {f"r{i}": seeded_tokens(n, cfg["vocab"], 50 * seed + i) for i, n in enumerate(lengths)}
    want = {rid: plain.forward(cfg, state, toks) for rid, toks in requests.items()}
    return folder, requests, want


def dev(values, dtype=torch.int32):
    return torch.tensor(values, dtype=dtype, device="cuda")


# ------------------------------------------------------------------------------------------------- kernels alone
@pytest.mark.parametrize("experts,top,groups,keep", [(10, 2, 5, 3), (8, 2, 4, 2), (6, 3, 1, 1), (4, 1, 2, 2), (9, 2, 3, 1), (64, 6, 8, 3),
                                                     (256, 8, 8, 4), (5, 5, 5, 5), (6, 2, 6, 2)])
def test_router_with_softmax_scores_and_groups(gpu, experts, top, groups, keep):
    """Against the plain rule on the same float32 logits; the logits ride in a wider buffer, as the part lays them out."""
    from stride_b200.csrc import ops
    g = torch.Generator().manual_seed(experts * top)
    tokens = 67
    logits = torch.zeros(tokens, experts + 3)
    logits[:, :experts] = torch.randn(tokens, experts, generator=g) * 2.0
    router = {"experts": experts, "top": top, "scale": 2.5, "groups": {"count": groups, "keep": keep}}
    want_ids, want_w = plain.route(logits[:, :experts].double(), {"p.router": torch.eye(experts, dtype=torch.float64)}, "p.", router)
    ids = torch.full((tokens + 1, top), -5, dtype=torch.int32, device="cuda")
    weights = torch.zeros(tokens + 1, top, device="cuda")
    seq = torch.zeros(tokens + 1, dtype=torch.int32, device="cuda")
    seq[-1] = -1
    ops.moe_select_groups(torch.cat([logits, logits[:1]]).cuda(), None, seq, ids, weights, experts, groups, keep, 2.5, softmax=True,
                          group_max=True, keep_scores=True)
    assert ids[:tokens].cpu().tolist() == want_ids
    close(weights[:tokens], torch.tensor([[float(a) for a in row] for row in want_w], dtype=torch.float64), 1e-5)
    assert ids[-1].cpu().tolist() == [-1] * top and float(weights[-1].abs().max()) == 0.0


def test_router_counts_a_group_by_its_best_member_and_does_not_renormalize(gpu):
    """Group 0 holds the single best expert, group 1 the two next best: by the sum of two members group 1 would win, by the
    best member group 0 does. The weights are the softmax scores themselves times the scale."""
    from stride_b200.csrc import ops
    logits = torch.tensor([[3.0, -4.0, -4.0, 2.5, 2.4, -4.0]])
    router = {"experts": 6, "top": 2, "scale": 1.5, "groups": {"count": 2, "keep": 1}}
    want_ids, want_w = plain.route(logits.double(), {"p.router": torch.eye(6, dtype=torch.float64)}, "p.", router)
    assert want_ids == [[0, 1]]
    ids, weights = torch.zeros(1, 2, dtype=torch.int32, device="cuda"), torch.zeros(1, 2, device="cuda")
    ops.moe_select_groups(logits.cuda(), None, None, ids, weights, 6, 2, 1, 1.5, softmax=True, group_max=True, keep_scores=True)
    assert ids.cpu().tolist() == want_ids
    close(weights, torch.tensor([[float(a) for a in row] for row in want_w], dtype=torch.float64), 1e-6)
    assert float(weights.sum()) < 1.0           # 1.5 * (0.43 + 0.0004): nothing was divided by the chosen scores' sum


@pytest.mark.parametrize("dtype,tol", [("float32", 1e-5), ("bfloat16", 2e-2)])
@pytest.mark.parametrize("width,ff,experts,top,tokens", [(96, 24, 8, 2, 37), (100, 14, 9, 2, 37), (128, 64, 4, 1, 37), (136, 72, 6, 3, 400),
                                                         (64, 128, 5, 2, 700)])
def test_silu_experts_and_the_gated_shared_expert(gpu, dtype, tol, width, ff, experts, top, tokens):
    """The routed feed-forward as a part against the plain mixture; steps of many rows run the experts on the tcgen05 tiles
    in bfloat16."""
    from stride_b200.config import FeedForwardSpec
    from stride_b200.parts import Runtime, build_part
    mlp = cases.moe(experts, top, ff, groups=None, scale=1.5, shared=ff + 6)
    cfg = cases.config(width, 50, [(cases.lstm(1, 8), mlp)])
    state = {k: v.to(STORED[dtype]) for k, v in cases.seeded_state(cfg, 5).items() if k.startswith("l0.mlp.")}
    rt = Runtime("cuda", STORED[dtype], max(64, tokens), 4)
    part = build_part("feed_forward", FeedForwardSpec("routed_experts", width, ff, "silu", "l0.mlp.", params=(
        ("experts", experts), ("top", top), ("router", "softmax_groups"), ("route_scale", 1.5), ("shared", ff + 6), ("shared_gate", True))), rt)
    assert set(part.declare()) == set(state)
    part.bind({k: (v.float() if v.dim() == 1 else v).cuda() for k, v in state.items()})
    for name, t in part.named_tensors().items():
        assert torch.equal(t.cpu().to(state[name].dtype), state[name]), name
    g = torch.Generator().manual_seed(width)
    x = (torch.randn(tokens, width, generator=g) * 1.5).to(STORED[dtype])

    class Ctx:
        seq_of_token = torch.zeros(max(64, tokens), dtype=torch.int32, device="cuda")
    out = part.forward(x.cuda(), Ctx)
    want = plain.feed_forward(x.double(), {k: v.double() for k, v in state.items()}, "l0.mlp.", mlp)
    close(out, want, tol)


@pytest.mark.parametrize("dtype,tol", [("float32", 3e-6), ("bfloat16", 1e-2)])
@pytest.mark.parametrize("nq,nkv,hd,vd,taps,normed", [(3, 1, 32, 32, 3, True), (4, 4, 16, 24, 4, True), (2, 2, 48, 16, 1, True), (3, 3, 20, 18, 2, True),
                                                      (2, 1, 128, 256, 16, True), (2, 2, 8, 8, 0, True), (2, 1, 16, 8, 5, False)])
def test_convolution_head_norms_cache_write_and_tails(gpu, dtype, tol, nq, nkv, hd, vd, taps, normed):
    """Three requests in one step (a start, a portion deep inside a request, a single token) against the plain convolution
    over each request's whole past; then the tails as the next step must find them."""
    from stride_b200.csrc import ops
    g = torch.Generator().manual_seed(hd + vd + taps)
    C = (nq + nkv) * hd + nkv * vd
    keep = max(taps - 1, 0)
    past, new = [0, 9, 1], [7, 5, 1]                        # tokens a request held before the step, and brings now
    page, pages = 4, 12
    histories = [(torch.randn(p + n, C, generator=g) * 2).to(STORED[dtype]) for p, n in zip(past, new)]
    raw = torch.cat([h[p:] for h, p in zip(histories, past)] + [torch.zeros(1, C, dtype=STORED[dtype])])       # one padded row
    tokens = raw.shape[0]
    conv_w = torch.randn(C, taps, generator=g) * 0.7 if taps else None
    wq, wk = (1.0 + 0.3 * torch.randn(hd, generator=g), 1.0 + 0.3 * torch.randn(hd, generator=g)) if normed else (None, None)
    slots_of_state = [2, 0, 1]
    state = torch.full((3, 5 + keep * C), float("nan"), device="cuda")
    for h, p, slot in zip(histories, past, slots_of_state):
        tail = torch.zeros(keep, C)
        if keep and p:
            rows = h[max(0, p - keep):p].float()
            tail[keep - rows.shape[0]:] = rows
        state[slot, 5:] = tail.reshape(-1).cuda()
    seq_of = dev([0] * new[0] + [1] * new[1] + [2] * new[2] + [-1])
    q_start, q_len = dev([0, new[0], new[0] + new[1], 0]), dev(new + [0])
    slot_map = torch.randperm(page * pages, generator=g)[:tokens].to(torch.int32)
    slot_map[-1] = -1
    k_pages = torch.full((pages, nkv, page, hd), 7.0, dtype=STORED[dtype], device="cuda")
    v_pages = torch.full((pages, nkv, page, vd), 7.0, dtype=STORED[dtype], device="cuda")
    out = torch.zeros(tokens, C + 8, dtype=STORED[dtype], device="cuda")
    ops.conv_head_norm(raw.cuda(), out, conv_w.t().contiguous().cuda() if taps else None, state if keep else None, 5, seq_of, q_start, dev(slots_of_state + [0]),
                       wq.cuda() if normed else None, wk.cuda() if normed else None, 1e-5, slot_map.cuda(), k_pages, v_pages, nq, nkv, hd, vd, page)
    if keep:
        ops.conv_tail(raw.cuda(), state, 5, q_start, q_len, dev(slots_of_state + [0]), 4, C, taps)
    at = 0
    for h, p, n, slot in zip(histories, past, new, slots_of_state):
        y = plain.short_convolution(h.double(), conv_w.double()) if taps else h.double()
        q = y[:, :nq * hd].view(-1, nq, hd)
        k = y[:, nq * hd:(nq + nkv) * hd].view(-1, nkv, hd)
        if normed:
            q, k = plain.rms_norm(q, wq.double(), 1e-5), plain.rms_norm(k, wk.double(), 1e-5)
        v = y[:, (nq + nkv) * hd:].view(-1, nkv, vd)
        want = torch.cat([q.reshape(-1, nq * hd), k.reshape(-1, nkv * hd), v.reshape(-1, nkv * vd)], dim=1)[p:]
        close(out[at:at + n, :C], want, tol)
        for r in range(n):
            s = int(slot_map[at + r])
            close(k_pages[s // page, :, s % page], k[p + r], tol)
            close(v_pages[s // page, :, s % page], v[p + r], tol)
        if keep:
            tail = torch.zeros(keep, C, dtype=torch.float64)
            rows = h[max(0, p + n - keep):].double()
            tail[keep - rows.shape[0]:] = rows
            assert torch.equal(state[slot, 5:].cpu().double(), tail.reshape(-1)), "the tail is the last projected rows, exactly"
        at += n
    assert float(out[-1].abs().max()) == 0.0            # the padded row is not touched


@pytest.mark.parametrize("dtype,tol", [("float32", 2e-5), ("bfloat16", 2e-5)])
@pytest.mark.parametrize("H,D,DV,cap", [(2, 24, 16, 6.0), (1, 8, 40, 20.0), (2, 64, 128, 12.0), (3, 10, 14, 4.0), (1, 256, 20, 8.0), (4, 16, 16, 2.0)])
def test_matrix_lstm_scan(gpu, dtype, tol, H, D, DV, cap):
    """Two requests with a past (their memories in the state rows) and a fresh one, against the recurrence token by token
    in float64 on the same inputs; then the state rows as the next step must find them. The inputs are the same numbers in
    both storage types (the scan itself is float32), so one bound holds."""
    from stride_b200.csrc import ops
    g = torch.Generator().manual_seed(H * D + DV)
    new, slots = [37, 1, 5], [1, 2, 0]
    tokens = sum(new) + 1
    ld = 2 * H * D + 2 * H * DV + 8
    k_off, v_off = H * D, 2 * H * D + 8
    proj = (torch.randn(tokens, ld, generator=g)).to(STORED[dtype])
    gates = torch.randn(tokens, 2 * H + 3, generator=g) * 3.0
    bias_i, bias_f = torch.randn(H, generator=g), 2.0 + torch.randn(H, generator=g)
    floats = H * D * DV + H * D + H
    state = torch.zeros(3, floats + 4)
    state[1, :H * D * DV + H * D] = torch.randn(H * D * DV + H * D, generator=g)       # a request with a past: S, n and m
    state[1, H * D * DV + H * D:floats] = torch.rand(H, generator=g) * 3.0
    state[2, :floats] = state[1, :floats] * 0.5
    state_dev = state.cuda()
    o = torch.full((tokens, H * DV), float("nan"), device="cuda")
    q_start = dev([0, new[0], new[0] + new[1], 0])
    ops.mlstm_scan(proj.cuda(), 0, k_off, v_off, gates.cuda(), bias_i.cuda(), bias_f.cuda(), cap, D ** -0.5, o, state_dev, q_start,
                   dev(new + [0]), dev(slots + [0]), 4, H, D, DV)
    at = 0
    for n, slot in zip(new, slots):
        x = proj[at:at + n].double()
        for a in range(H):
            S = state[slot, a * D * DV:(a + 1) * D * DV].double().view(D, DV).clone()
            nn = state[slot, H * D * DV + a * D:H * D * DV + (a + 1) * D].double().clone()
            top = float(state[slot, H * D * DV + H * D + a])
            for t in range(n):
                q, k, v = x[t, a * D:(a + 1) * D] * D ** -0.5, x[t, k_off + a * D:k_off + (a + 1) * D], x[t, v_off + a * DV:v_off + (a + 1) * DV]
                li = cap * math.tanh((float(gates[at + t, a]) + float(bias_i[a])) / cap)
                lf = plain.log_sigmoid(cap * math.tanh((float(gates[at + t, H + a]) + float(bias_f[a])) / cap))
                new_top = max(lf + top, li)
                keep, take = math.exp(lf + top - new_top), math.exp(li - new_top)
                S, nn, top = keep * S + take * torch.outer(k, v), keep * nn + take * k, new_top
                want = (S.T @ q) / (max(abs(float(nn @ q)), math.exp(-top)) + 1e-6)
                got = o[at + t, a * DV:(a + 1) * DV].double().cpu()
                assert float((got - want).abs().max()) <= tol * max(1.0, float(want.abs().max())), f"request {slot}, head {a}, token {t}"
            close(state_dev[slot, a * D * DV:(a + 1) * D * DV], S.reshape(-1), 1e-5)
            close(state_dev[slot, H * D * DV + a * D:H * D * DV + (a + 1) * D], nn, 1e-5)
            assert abs(float(state_dev[slot, H * D * DV + H * D + a]) - top) <= 1e-5 * max(1.0, abs(top))
        at += n
    assert torch.equal(state_dev[:, floats:].cpu(), state[:, floats:])      # nothing beyond a row's memory is touched


@pytest.mark.parametrize("H,D,DV,cap,ld_pad", [(2, 24, 16, 6.0, 0), (1, 128, 136, 15.0, 0), (3, 10, 14, 4.0, 3), (1, 200, 20, 15.0, 0)])
def test_matrix_lstm_chunks(gpu, H, D, DV, cap, ld_pad):
    """Long portions chunk by chunk (one chunk, whole and broken ones, more than the 256 tokens of a turn of the gates' scan; with a past
    and fresh): no further from the recurrence in float64 than the chain of tokens (half as much again is left for the luck of the
    draw), in outputs and in the state rows."""
    from stride_b200.csrc import ops
    g = torch.Generator().manual_seed(H * D + DV)
    new, slots = [130, 64, 289, 1], [1, 2, 0, 3]
    tokens = sum(new) + 1
    k_off, v_off = H * D, 2 * H * D + 8
    ld = v_off + H * DV + ld_pad
    proj = torch.randn(tokens, ld, generator=g).bfloat16()
    gates = torch.randn(tokens, 2 * H + 3, generator=g) * 2.0
    bias_i, bias_f = torch.randn(H, generator=g), 2.0 + torch.randn(H, generator=g)
    floats = H * D * DV + H * D + H
    state = torch.zeros(4, (floats + 7) // 4 * 4)
    state[1, :H * D * DV + H * D] = torch.randn(H * D * DV + H * D, generator=g)
    state[1, H * D * DV + H * D:floats] = torch.rand(H, generator=g) * 3.0
    state[2, :floats] = state[1, :floats] * 0.5
    want, want_state, at = torch.zeros(tokens - 1, H * DV, dtype=torch.float64), state.double().clone(), 0
    for n, slot in zip(new, slots):
        x = proj[at:at + n].double()
        for a in range(H):
            S = state[slot, a * D * DV:(a + 1) * D * DV].double().view(D, DV).clone()
            nn = state[slot, H * D * DV + a * D:H * D * DV + (a + 1) * D].double().clone()
            top = float(state[slot, H * D * DV + H * D + a])
            for t in range(n):
                q, k, v = x[t, a * D:(a + 1) * D] * D ** -0.5, x[t, k_off + a * D:k_off + (a + 1) * D], x[t, v_off + a * DV:v_off + (a + 1) * DV]
                li = cap * math.tanh((float(gates[at + t, a]) + float(bias_i[a])) / cap)
                lf = plain.log_sigmoid(cap * math.tanh((float(gates[at + t, H + a]) + float(bias_f[a])) / cap))
                new_top = max(lf + top, li)
                keep, take = math.exp(lf + top - new_top), math.exp(li - new_top)
                S, nn, top = keep * S + take * torch.outer(k, v), keep * nn + take * k, new_top
                want[at + t, a * DV:(a + 1) * DV] = (S.T @ q) / (max(abs(float(nn @ q)), math.exp(-top)) + 1e-6)
            want_state[slot, a * D * DV:(a + 1) * D * DV] = S.reshape(-1)
            want_state[slot, H * D * DV + a * D:H * D * DV + (a + 1) * D] = nn
            want_state[slot, H * D * DV + H * D + a] = top
        at += n
    results = []
    for chunks in (False, True):
        state_dev, o = state.cuda(), torch.full((tokens, H * DV), float("nan"), device="cuda")
        args = (proj.cuda(), 0, k_off, v_off, gates.cuda(), bias_i.cuda(), bias_f.cuda(), cap, D ** -0.5, o, state_dev,
                dev([0, new[0], new[0] + new[1], sum(new[:3]), 0]), dev(new + [0]), dev(slots + [0]), 5, H, D, DV)
        if chunks:
            scratch = torch.full((ops.mlstm_chunks_scratch_floats(5, max(new), H, D, DV),), float("nan"), device="cuda")
            ops.mlstm_chunks(*args, max(new), scratch)
        else:
            ops.mlstm_scan(*args)
        assert bool(o[-1].isnan().all()) and torch.equal(state_dev[:, floats:].cpu(), state[:, floats:])
        error = lambda x, y: float((x.double().cpu() - y).norm() / y.norm())
        results.append((error(o[:-1], want), error(state_dev[:, :floats], want_state[:, :floats])))
    assert all(c <= 1.5 * r + 2.0 ** -24 and r < 1e-4 for r, c in zip(*results)), results


@pytest.mark.parametrize("dtype,tol", [("float32", 3e-6), ("bfloat16", 1e-2)])
def test_latent_norm_between_two_products(gpu, dtype, tol):
    from stride_b200.csrc import ops
    g = torch.Generator().manual_seed(3)
    for width, offset, ld in ((24, 0, 40), (10, 8, 30), (96, 16, 200), (50, 2, 64)):
        x = (torch.randn(9, ld, generator=g) * 3).to(STORED[dtype])
        w = 1.0 + 0.3 * torch.randn(width, generator=g)
        out = torch.zeros(9, width, dtype=STORED[dtype], device="cuda")
        ops.rms_norm_cols(x.cuda(), offset, width, w.cuda(), out, 1e-4)
        close(out, plain.rms_norm(x[:, offset:offset + width].double(), w.double(), 1e-4), tol)


@pytest.mark.parametrize("dtype,tol", [("float32", 1e-5), ("bfloat16", 1.5e-2)])
@pytest.mark.parametrize("heads,rank,rot,page", [(3, 40, 8, 8), (6, 64, 16, 16), (2, 18, 6, 4), (16, 128, 32, 16)])
def test_latent_attention_with_sinks(gpu, dtype, tol, heads, rank, rot, page):
    """Portions and single tokens over latent pages with a sink per head, one of them far above every score: the exact
    kernel in both types, and the tensor-core kernels (portions; single tokens with the keys split) where they take the sizes."""
    from stride_b200.csrc import ops
    g = torch.Generator().manual_seed(heads * rank)
    lens = [(0, 70), (40, 9), (130, 1), (257, 1)]
    total_pages = sum(-(-(c + n) // page) for c, n in lens) + 2
    perm = torch.randperm(total_pages, generator=g).tolist()
    table = torch.zeros(len(lens), max(-(-(c + n) // page) for c, n in lens), dtype=torch.int32)
    q_start, q_len, ctx_len, seq_of, positions, at = [], [], [], [], [], 0
    for s, (c, n) in enumerate(lens):
        pages = [perm.pop() for _ in range(-(-(c + n) // page))]
        table[s, :len(pages)] = torch.tensor(pages)
        q_start.append(at), q_len.append(n), ctx_len.append(c + n)
        seq_of += [s] * n
        positions += list(range(c, c + n))
        at += n
    tokens = at
    lat = (torch.randn(total_pages, 1, page, rank, generator=g)).to(STORED[dtype])
    kr = (torch.randn(total_pages, 1, page, rot, generator=g)).to(STORED[dtype])
    qa = (torch.randn(tokens, heads * (rank + rot), generator=g) * 0.5).to(STORED[dtype])
    sinks = torch.randn(heads, generator=g)
    sinks[0] = 9.0
    scale = 0.3
    want = torch.zeros(tokens, heads, rank, dtype=torch.float64)
    for t in range(tokens):
        s, pos = seq_of[t], positions[t]
        rows = lambda cache: torch.stack([cache[int(table[s, j // page]), 0, j % page] for j in range(pos + 1)]).double()
        c, k = rows(lat), rows(kr)
        for a in range(heads):
            q = qa[t, a * (rank + rot):(a + 1) * (rank + rot)].double()
            sc = (c @ q[:rank] + k @ q[rank:]) * scale
            e = torch.exp(sc - sc.max())
            want[t, a] = (e[:, None] * c).sum(0) / (e.sum() + math.exp(float(sinks[a]) - float(sc.max())))
    want = want.reshape(tokens, heads * rank)
    got = torch.zeros(tokens, heads * rank, dtype=STORED[dtype], device="cuda")
    args = (lat.cuda(), kr.cuda(), table.cuda())
    ops.latent_attention(qa.cuda(), got, *args, dev(seq_of), dev(positions), heads, rank, rot, page, scale, sinks=sinks.cuda())
    close(got, want, tol)
    without = torch.zeros_like(got)
    ops.latent_attention(qa.cuda(), without, *args, dev(seq_of), dev(positions), heads, rank, rot, page, scale)
    assert float((without.double().cpu() - want).abs().max()) > 0.05, "the sinks do not show in this case"
    if not ops.latent_tc_supported(STORED[dtype], heads, rank, rot):
        return
    fast = torch.full((tokens, heads * rank), float("nan"), dtype=torch.bfloat16, device="cuda")
    split = 79
    ops.latent_attention_tc(qa.cuda(), fast, None, *args, dev(q_start), dev(q_len), dev(ctx_len), dev(seq_of), 0, 2, 0, split, 70, heads, rank, rot,
                            page, scale, sinks=sinks.cuda())
    for splits, per in ((1, 0), (3, 128)):
        partial = torch.zeros(tokens * heads * splits * (rank + 2), device="cuda") if splits > 1 else None
        ops.latent_attention_tc(qa.cuda(), fast, partial, *args, dev(q_start), dev(q_len), dev(ctx_len), dev(seq_of), 2, 2, split, 2, 1, heads, rank,
                                rot, page, scale, splits=splits, keys_per_split=per, sinks=sinks.cuda())
        torch.cuda.synchronize()
        close(fast, want, 2e-2)


@pytest.mark.parametrize("dtype,tol", [("float32", 1e-5), ("bfloat16", 1.5e-2)])
def test_the_input_of_a_pass(gpu, dtype, tol):
    """x <- W [x; x0] + s[t] through the part, for a pass in the middle."""
    from stride_b200.config import PassInputSpec
    from stride_b200.parts import ResidualStream, Runtime, build_part
    for width, tokens in ((40, 5), (100, 23), (256, 70)):
        rt = Runtime("cuda", STORED[dtype], 128, 4)
        g = torch.Generator().manual_seed(width)
        part = build_part("pass_input", PassInputSpec("mix_embedding", width, 3, "loop.in", "loop.step"), rt)
        assert {k: v.shape for k, v in part.declare().items()} == {"loop.in": (width, 2 * width), "loop.step": (3, width)}
        w = (torch.randn(width, 2 * width, generator=g) / math.sqrt(2 * width)).to(STORED[dtype])
        steps = torch.randn(3, width, generator=g)
        part.bind({"loop.in": w.cuda(), "loop.step": steps.cuda()})
        x, x0 = torch.randn(tokens, width, generator=g), torch.randn(tokens, width, generator=g).to(STORED[dtype])
        stream = ResidualStream(rt, tokens, width)
        stream.residual.copy_(x)

        class Ctx:
            seq_of_token = torch.zeros(128, dtype=torch.int32, device="cuda")
        part.forward(stream, x0.cuda(), 1, Ctx)
        seen = x.to(STORED[dtype]).double()                 # the product reads the stream in the compute dtype
        close(stream.materialize(), torch.cat([seen, x0.double()], dim=1) @ w.double().T + steps[1].double(), tol)


def test_scaled_output_norm(gpu):
    """x += s * w * unit_rms(y): the learned scale is a param of the norm on a sublayer's output."""
    from stride_b200.config import NormSpec
    from stride_b200.parts import ResidualStream, Runtime, build_part
    for width in (54, 64, 1032):
        rt = Runtime("cuda", torch.float32, 16, 4)
        g = torch.Generator().manual_seed(width)
        norm = build_part("norm", NormSpec("rmsnorm", width, 1e-3, "n", (("tensor", "n"), ("scale_tensor", "s"))), rt)
        w, s = 1.0 + 0.3 * torch.randn(width, generator=g), 0.5 + 0.3 * torch.randn(width, generator=g)
        norm.bind({"n": w.cuda(), "s": s.cuda()})
        assert torch.equal(norm.named_tensors()["n"].cpu(), w) and torch.equal(norm.named_tensors()["s"].cpu(), s)
        x, y = torch.randn(6, width, generator=g), torch.randn(6, width, generator=g) * 5
        stream = ResidualStream(rt, 6, width)
        stream.residual.copy_(x)
        stream.add_normed(y.cuda(), norm, 1.0, keep_copy=False)
        want = x.double() + plain.rms_norm(y.double(), w.double(), 1e-3) * s.double()
        close(stream.materialize(), want, 3e-6)
        # left for the next norm, the sum and that norm are one kernel; asked for rows only, the sum runs alone first
        front = build_part("norm", NormSpec("rmsnorm", width, 1e-5, "f", (("tensor", "f"),)), rt)
        front.bind({"f": (w * 0.5 + 0.2).cuda()})
        stream.add_normed(y.cuda(), norm, 0.5, keep_copy=False)
        want = want + 0.5 * plain.rms_norm(y.double(), w.double(), 1e-3) * s.double()
        close(stream.normed(front), plain.rms_norm(want, (w * 0.5 + 0.2).double(), 1e-5), 3e-6)
        close(stream.materialize(), want, 3e-6)
        stream.add_normed(y.cuda(), norm, -0.25, keep_copy=False)
        want = want - 0.25 * plain.rms_norm(y.double(), w.double(), 1e-3) * s.double()
        close(stream.normed(front, rows=torch.tensor([4, 1], dtype=torch.int32, device="cuda")),
              plain.rms_norm(want[[4, 1]], (w * 0.5 + 0.2).double(), 1e-5), 3e-6)
        close(stream.materialize(), want, 3e-6)


# ------------------------------------------------------------------- each mechanism in a model of nothing else
ONLY_LATENT = cases.config(72, 101, [(cases.latent(3, 12, 8, 10, 24, 16, scale=0.5, scaling=(3.0, 32, 4.0, 1.0)), None),
                                     (cases.latent(1, 6, 2, 20, 8, 30, scale=0.8), None)])
ONLY_WINDOWED = cases.config(56, 89, [(cases.windowed(3, 1, 12, 8, conv=3, window=9, softcap=4.0, scale=0.9), None),
                                      (cases.windowed(2, 2, 8, 12, conv=5, scale=0.5), None)])
ONLY_LSTM = cases.config(48, 67, [(cases.lstm(2, 12, 20, cap=5.0), None), (cases.lstm(1, 40, 8, cap=15.0), None)])
ONLY_FF = cases.config(56, 89, [(cases.lstm(1, 4), cases.dense(70)), (cases.lstm(1, 4), cases.moe(10, 2, 10, groups=(5, 3), scale=1.3, shared=18)),
                                (cases.lstm(1, 4), cases.moe(5, 1, 6, scale=3.0))])
ONLY_LOOP = cases.config(40, 53, [(cases.lstm(1, 8), None), (cases.lstm(1, 8), None)], loop=(1, 2, 4))


@pytest.mark.parametrize("name,cfg", [("latent", ONLY_LATENT), ("windowed", ONLY_WINDOWED), ("lstm", ONLY_LSTM), ("ff", ONLY_FF), ("loop", ONLY_LOOP)])
def test_each_mechanism_in_a_model_of_its_own(gpu, tmp_models, name, cfg):
    folder, requests, want = model_case(tmp_models, name, cfg, "float32", 7, [45, 19, 3])
    replay(folder, "float32", modes.whole(requests), want, 8, 2, name + " whole")
    replay(folder, "float32", modes.changing_portions(requests), want, 8, 2, name + " portions")
    replay(folder, "float32", modes.tail_one_by_one(requests, tail=15), want, 8, 2, name + " decode")


@pytest.mark.parametrize("case", ["A", "C"])
def test_the_stream_after_every_layer_run(gpu, tmp_models, case):
    """Run by run in float32: the first run that differs names the mechanism."""
    from stride_b200.engine.trace import TraceSession
    cfg = cases.CASES[case]
    state = cases.seeded_state(cfg, 3)
    folder = write_model_dir(str(tmp_models / f"netusun_layers_{case}"), cfg, state, torch.float32)
    tokens = seeded_tokens(29, cfg["vocab"], 4)
    want = []
    plain.forward(cfg, {k: v.double() for k, v in state.items()}, tokens, capture=want)
    session = TraceSession(folder, "float32", max_tokens=64, block_size=8, max_requests=1)
    session.model.capture = []
    session.run_step({"step": 0, "entries": [{"id": "a", "tokens": tokens, "want": [0]}], "end": ["a"]})
    assert len(session.model.capture) == len(want) == cases.run_count(cfg)
    for i, (got, expected) in enumerate(zip(session.model.capture, want)):
        err = float((got.double().cpu() - expected).abs().max())
        assert err <= 2e-5 * float(expected.abs().max()), f"the stream differs after run {i}: {err:.3e}"


# ---------------------------------------------------------------------------- whole models, every cutting
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("case,page", [("A", 16), ("B", 8), ("C", 16), ("D", 32)])
def test_every_cutting_gives_the_plain_logits(gpu, tmp_models, case, page, dtype):
    cfg = cases.CASES[case]
    folder, requests, want = model_case(tmp_models, case, cfg, dtype, 11, [90, 33, 1, 52, 9, 2])
    # bfloat16: a router's close call may fall the other way on rounded activations, which changes a row outright
    share = 1.0 if dtype == "float32" else 0.9
    bound = BF16_BOUND_DEEP if case == "C" else BF16_BOUND
    replay(folder, dtype, modes.whole(requests), want, page, 2, "whole", min_ok=share, bound=bound)
    session = replay(folder, dtype, modes.tail_one_by_one(requests, tail=40), want, page, 2, "decode", min_ok=share, bound=bound)
    assert session.runner.graph_replays > 0, "single-token steps did not go through captured graphs"
    replay(folder, dtype, modes.changing_portions(requests), want, page, 2, "portions", min_ok=share, bound=bound)
    # three live requests, six requests in all: pages and state slots are used again
    replay(folder, dtype, modes.mixed(requests, live_limit=3, seed=5), want, page, 3, "mixed", min_ok=share, bound=bound)
    replay(folder, dtype, modes.decoding_together(dict(list(requests.items())[:4]), decode_steps=6, prompts_per_step=2), want, page, 4,
           "decoding together", min_ok=share, bound=bound)


def test_float32_logits_do_not_depend_on_the_cutting(gpu, tmp_models):
    """Bitwise: every sum of the 32-bit path has an order that depends on the token's position only."""
    from stride_b200.engine.trace import TraceSession
    folder, requests, _want = model_case(tmp_models, "bitwise", cases.CASE_A, "float32", 13, [41, 18, 27])
    results = []
    for steps in (modes.whole(requests), modes.changing_portions(requests), modes.mixed(requests, live_limit=3, seed=2)):
        session = TraceSession(folder, "float32", max_tokens=modes.peak_tokens(steps), block_size=8, max_requests=3)
        got = {}
        rows = modes.expected_rows(steps)
        for s in steps:
            out = session.run_step(s)
            for r, key in enumerate(rows[s["step"]]):
                got[key] = out[r].clone()
        results.append(got)
    for other in results[1:]:
        for key in other:
            assert torch.equal(other[key], results[0][key]), f"request {key[0]} position {key[1]} differs between cuttings"


# ------------------------------------------------------------------------ windows, far keys, long memories
def window_model(window, taps=2):
    """Two windowed layers with sharp scores (normed queries and keys at a scale of 2): single keys decide, so a window that
    is one key too short or too long changes the logits outright."""
    return cases.config(64, 61, [(cases.windowed(4, 2, 8, 8, conv=taps, window=window, softcap=30.0, scale=2.0), None),
                                 (cases.windowed(2, 1, 16, 8, conv=taps, window=window + 5, softcap=30.0, scale=1.5), cases.dense(32))])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("window,page", [(24, 8), (17, 4), (32, 16)])
def test_keys_at_a_windows_edge(gpu, tmp_models, dtype, window, page):
    """The plain logits of windows one key shorter and one key longer differ outright at the compared positions, in the
    prompt and among decoded tokens; the engine gives the design's. Windows that end on a page border and inside a page."""
    cfg = window_model(window)
    state = {k: v.double() for k, v in rounded(cases.seeded_state(cfg, 41), dtype).items()}
    tokens = seeded_tokens(130, cfg["vocab"], 8)
    full = plain.forward(cfg, state, tokens)
    for other in (window - 1, window + 1):
        off = plain.forward(window_model(other), state, tokens)
        moved = (off - full).abs().amax(dim=1) > 0.02 * full.abs().max()
        assert not moved[:min(window - 1, other)].any() and moved[window + 6:].sum() >= 40, "the window's edge does not show in these logits"
    folder = write_model_dir(str(tmp_models / f"netusun_window_{window}_{dtype}"), cfg, {k: v.float() for k, v in state.items()}, STORED[dtype])
    requests, want = {"w": tokens}, {"w": full}
    share = 1.0 if dtype == "float32" else 0.9
    replay(folder, dtype, modes.whole(requests), want, page, 1, "window whole", min_ok=share)
    replay(folder, dtype, modes.tail_one_by_one(requests, tail=80), want, page, 1, "window decode", min_ok=share)
    replay(folder, dtype, modes.changing_portions(requests, sizes=(7, 2, 33, 9, 2, 40)), want, page, 1, "window portions", min_ok=share)


def test_the_softmax_has_one_more_term(gpu, tmp_models):
    """Without the one in the denominator a head whose scores are all far below zero would still return a whole value; the
    design all but silences it. (A common factor on all heads would vanish in the norm that follows; heads that differ do
    not.) The plain logits without the term differ by a hundred times the float32 bound and more, most for the first tokens."""
    cfg = window_model(12)
    state = {k: v.double() for k, v in cases.seeded_state(cfg, 43).items()}
    tokens = seeded_tokens(40, cfg["vocab"], 3)
    full = plain.forward(cfg, state, tokens)
    original = plain.MIXERS["attention"]
    try:
        plain.MIXERS["attention"] = _window_attention_plain_softmax
        off = plain.forward(cfg, state, tokens)
    finally:
        plain.MIXERS["attention"] = original
    moved = (off - full).abs().amax(dim=1) / full.abs().max()
    assert (moved > 0.01).sum() >= 20 and moved[0] > 0.1
    folder = write_model_dir(str(tmp_models / "netusun_one_more"), cfg, {k: v.float() for k, v in state.items()}, torch.float32)
    replay(folder, "float32", modes.whole({"s": tokens}), {"s": full}, 4, 1, "one more term, whole")
    replay(folder, "float32", modes.tail_one_by_one({"s": tokens}, tail=30), {"s": full}, 4, 1, "one more term, decode")


def _window_attention_plain_softmax(h, w, p, m, eps):
    """The windowed mixer with an ordinary softmax (nothing added to the denominator): a negative control."""
    T = h.shape[0]
    H, G, D, DV = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (plain.short_convolution(h @ w[p + n].T, w[p + n + ".conv"]) for n in "qkv")
    q = plain.rms_norm(q.view(T, H, D), w[p + "q.norm"], eps)
    k = plain.rms_norm(k.view(T, G, D), w[p + "k.norm"], eps)
    v = v.view(T, G, DV)
    heads = torch.zeros(T, H, DV, dtype=torch.float64)
    for a in range(H):
        for i in range(T):
            first = max(0, i - m["mask"]["size"] + 1)
            s = m["softcap"] * torch.tanh((k[first:i + 1, a // (H // G)] * q[i, a]).sum(-1) * m["scale"] / m["softcap"])
            heads[i, a] = torch.softmax(s, 0) @ v[first:i + 1, a // (H // G)]
    return heads.reshape(T, H * DV) @ w[p + "o"].T


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_far_past_shows_through_sharp_latent_attention(gpu, tmp_models, dtype):
    """Scores sharp enough for single keys to decide, hundreds of tokens back: another far past (positions 0 .. 23 only)
    moves the plain logits beyond position 300, and the engine follows the true past, whole, decoded and in portions."""
    cfg = cases.config(64, 61, [(cases.latent(8, 8, 8, 8, 32, 16, scale=2.5, scaling=(2.0, 128, 16.0, 1.0)), None)])
    state = {k: v.double() for k, v in rounded(cases.seeded_state(cfg, 41), dtype).items()}
    for name in [n for n in state if n.endswith("sink")]:
        state[name] = state[name] - 3.0                     # sinks that leave the keys their say
    tokens = seeded_tokens(420, cfg["vocab"], 8)
    full = plain.forward(cfg, state, tokens)
    other = list(tokens)
    other[:24] = seeded_tokens(24, cfg["vocab"], 9)
    moved = (plain.forward(cfg, state, other) - full)[300:].abs().amax(dim=1) > 0.02 * full.abs().max()
    assert moved.sum() >= 20, "the far past does not show in these logits"
    folder = write_model_dir(str(tmp_models / f"netusun_far_{dtype}"), cfg, {k: v.float() for k, v in state.items()}, STORED[dtype])
    requests, want = {"far": tokens}, {"far": full}
    share = 1.0 if dtype == "float32" else 0.9
    keep = {"far": set(range(0, 420, 5)) | set(range(300, 420)) | {0, 1, 2, 3, 7, 8, 9, 15, 16, 17}}
    for page in (8, 16):
        replay(folder, dtype, modes.restrict_wants(modes.whole(requests), keep), want, page, 1, "far whole", min_ok=share)
        replay(folder, dtype, modes.tail_one_by_one(requests, tail=110), want, page, 1, "far decode", min_ok=share)
        replay(folder, dtype, modes.restrict_wants(modes.changing_portions(requests, sizes=(7, 2, 64, 9, 33, 2, 120)), keep), want, page, 1,
               "far portions", min_ok=share)


def test_a_memory_that_carries_its_first_tokens_over_hundreds_of_steps(gpu, tmp_models):
    """Forget gates close to one, and an input gate that opens for one token of the vocabulary only (its row of the input
    gate's matrix points along that token's normed embedding, the bias closes the gate for all others): the memory is that
    token's key and value, and another token in its place (position 3) moves the plain logits 400 steps later. The engine
    carries the memory through portions and single tokens, and a second request finds its slot cleared."""
    cfg = cases.config(48, 67, [(cases.lstm(2, 16, 24, cap=15.0), cases.dense(40))])
    state = {k: v.double() for k, v in cases.seeded_state(cfg, 19, forget_bias=9.0).items()}
    state["l0.mix.f"] = state["l0.mix.f"] * 0.1           # the forget gate hardly depends on the token
    special = 5
    seen = plain.rms_norm(state["embed"][special], state["l0.norm1"], cfg["norm"]["eps"])
    state["l0.mix.i"] = (40.0 * seen / (seen @ seen)).repeat(2, 1)
    state["l0.mix.i.b"] = torch.full((2,), -20.0, dtype=torch.float64)
    tokens = [t if t != special else special + 1 for t in seeded_tokens(430, cfg["vocab"], 8)]
    tokens[3] = special
    full = plain.forward(cfg, state, tokens)
    other = list(tokens)
    other[3] = special + 1
    moved = (plain.forward(cfg, state, other) - full)[400:].abs().amax(dim=1) > 0.05 * full.abs().max()
    assert moved.sum() >= 25, "the token at position 3 does not show in these logits"
    folder = write_model_dir(str(tmp_models / "netusun_memory"), cfg, {k: v.float() for k, v in state.items()}, torch.float32)
    second = seeded_tokens(60, cfg["vocab"], 10)
    requests, want = {"long": tokens, "next": second}, {"long": full, "next": plain.forward(cfg, state, second)}
    keep = {"long": set(range(0, 430, 7)) | set(range(395, 430)), "next": set(range(60))}
    replay(folder, "float32", modes.restrict_wants(modes.whole(requests), keep), want, 8, 1, "memory whole")
    replay(folder, "float32", modes.restrict_wants(modes.changing_portions(requests, sizes=(64, 2, 9, 120, 3)), keep), want, 8, 1, "memory portions")
    replay(folder, "float32", modes.tail_one_by_one(requests, tail=45), want, 8, 1, "memory decode")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_sharp_attention_and_long_decoding_on_the_tensor_core_sizes(gpu, tmp_models, dtype):
    """Head sizes 64 and 128 and a latent of 64 + 16 (what the tensor-core kernels take) without experts, whose close calls
    would hide what is looked for here: scores half as sharp again and 120 tokens decoded one by one, past both windows and
    across many page borders."""
    c = cases.CASE_C["layers"]
    cfg = cases.sharpened(cases.config(128, 263, [((c[0]["type"], c[0]["mixer"]), cases.dense(96)), ((c[1]["type"], c[1]["mixer"]), cases.dense(64)),
                                                  ((c[3]["type"], c[3]["mixer"]), None)], eps=2e-6), 1.5)
    folder, requests, want = model_case(tmp_models, "sharp", cfg, dtype, 17, [389, 131])
    share = 1.0 if dtype == "float32" else 0.9
    keep = {"r0": set(range(0, 389, 7)) | set(range(260, 389)) | {0, 1, 2, 3, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65}, "r1": set(range(0, 131, 3))}
    replay(folder, dtype, modes.restrict_wants(modes.whole(requests), keep), want, 16, 2, "whole", min_ok=share, bound=BF16_BOUND_DEEP)
    replay(folder, dtype, modes.restrict_wants(modes.changing_portions(requests, sizes=(7, 2, 64, 9, 33, 2, 120)), keep), want, 16, 2,
           "portions", min_ok=share, bound=BF16_BOUND_DEEP)
    replay(folder, dtype, modes.tail_one_by_one(requests, tail=120), want, 16, 2, "long decode", min_ok=share, bound=BF16_BOUND_DEEP)


# --------------------------------------------------------------------------- generation through the engine
def test_greedy_generation_through_the_engine(gpu, tmp_models):
    from stride_b200 import Engine, SamplingParams
    cfg = cases.CASE_A
    state = cases.seeded_state(cfg, 29)
    folder = write_model_dir(str(tmp_models / "netusun_generate"), cfg, state, torch.float32)
    state = {k: v.double() for k, v in state.items()}
    prompts = [seeded_tokens(n, cfg["vocab"], 300 + n) for n in (37, 5, 18, 1, 26)]
    new = 9
    expected = []
    for prompt in prompts:
        seq = list(prompt)
        for _ in range(new):
            seq.append(int(plain.forward(cfg, state, seq)[-1].argmax()))
        expected.append(seq[len(prompt):])
    # a token budget below the longest prompt: prompts go in portions beside the others' decoded tokens
    engine = Engine(folder, dtype="float32", block_size=8, num_blocks=64, max_batch_tokens=16, max_batch_seqs=3, max_model_len=64,
                    check_invariants=True)
    outs = engine.generate(copy.deepcopy(prompts), SamplingParams(temperature=0.0, max_tokens=new, ignore_eos=True))
    assert [o.tokens for o in outs] == expected


def lstm_case(H, D, DV, lens, seed):
    """Projections and gates as a model's products make them, the arguments of the scan for them from empty memories, and the float64
    outputs [tokens, H, DV]."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    tokens, floats = sum(lens), H * D * DV + H * D + H
    proj = (torch.randn(tokens, 2 * H * D + H * DV, generator=g, device="cuda") * 0.9).bfloat16()
    gates = torch.randn(tokens, 2 * H, generator=g, device="cuda") * 0.9
    bias, cap, want, at = torch.ones(H, device="cuda"), 15.0, [], 0
    for n in filter(None, lens):
        x = proj[at:at + n].double()
        q, k, v = x[:, :H * D].view(n, H, D) * D ** -0.5, x[:, H * D:2 * H * D].view(n, H, D), x[:, 2 * H * D:].view(n, H, DV)
        li, f = (cap * torch.tanh((z.double() + 1.0) / cap) for z in (gates[at:at + n, :H], gates[at:at + n, H:]))
        lf = torch.nn.functional.logsigmoid(f)
        b, m, tops = torch.cumsum(lf, 0), torch.zeros(H, dtype=torch.float64, device="cuda"), []
        for t in range(n):
            m = torch.maximum(lf[t] + m, li[t])
            tops.append(m)
        tops = torch.stack(tops)
        w = (b[:, None] - b[None, :] + li[None, :] - tops[:, None]).masked_fill(torch.triu(torch.ones(n, n, dtype=torch.bool, device="cuda"), 1)[..., None], float("-inf")).exp()
        s = torch.einsum("ihd,jhd->ijh", q, k) * w
        want.append(torch.einsum("ijh,jhv->ihv", s, v) / (torch.maximum(s.sum(1).abs(), torch.exp(-tops)) + 1e-6)[..., None])
        at += n
    starts = [sum(lens[:i]) for i in range(len(lens))]

    def run(records=None, chunks=True):
        from stride_b200.csrc import ops
        state, o = torch.zeros(len(lens), floats, device="cuda"), torch.full((tokens, H * DV), float("nan"), device="cuda")
        args = (proj, 0, H * D, 2 * H * D, gates, bias, bias, cap, D ** -0.5, o, state, dev(starts), dev(lens), dev(list(range(len(lens)))), len(lens), H, D, DV)
        if chunks:
            scratch = torch.full((ops.mlstm_chunks_scratch_floats(len(lens), max(lens), H, D, DV, records),), float("nan"), device="cuda")
            ops.mlstm_chunks(*args, max(lens), scratch, records)
        else:
            ops.mlstm_scan(*args)
        return o, state

    return run, torch.cat(want)


@pytest.mark.parametrize("H,D,DV,lens", [(8, 128, 128, [500]), (8, 128, 128, [96, 130]), (4, 256, 128, [200]), (6, 100, 72, [300, 64])])
def test_matrix_lstm_chunks_are_no_further_from_float64_than_the_chain(gpu, H, D, DV, lens):
    """The median over a step's (token, head) rows, which single rows whose divisor all but vanishes do not move (over 16 seeds the
    ratio lay within 0.72 and 0.92)."""
    run, want = lstm_case(H, D, DV, lens, 5)
    error = lambda o: float(((o.double().view(want.shape) - want).norm(dim=-1) / want.norm(dim=-1)).median())
    assert error(run()[0]) <= error(run(chunks=False)[0])


def test_matrix_lstm_chunks_lie_close(gpu):
    """A long portion beside short and empty ones: room for the chunks that there are, and the same bits in it as in one with a long
    portion's chunks for every request."""
    from stride_b200.csrc import ops
    lens = [7, 130, 1, 64, 0, 5, 200, 65, 0]
    run, _want = lstm_case(3, 24, 16, lens, 9)
    records = sum(-(-n // ops.DECAY_CHUNK) for n in lens)
    whole, close_by = run(), run(records)
    assert torch.equal(whole[0], close_by[0]) and torch.equal(whole[1], close_by[1])
    assert not bool(whole[0].isnan().any())
    spread, packed = (ops.mlstm_chunks_scratch_floats(201, 1000, 16, 128, 128, r) * 4 for r in (None, 216))
    assert packed < 0.26e9 < 3.5e9 < spread


def test_matrix_lstm_takes_the_chunks_where_they_pay_and_fit(gpu):
    """One long portion beside many short ones stays token by token, as do steps whose chunks would need more room than allowed."""
    from types import SimpleNamespace

    from stride_b200.parts.mlstm import MatrixLstmMixer
    part = SimpleNamespace(H=16, D=128, DV=128, _room=MatrixLstmMixer._room)

    def chunks(lens, given=True):
        ctx = SimpleNamespace(decode_tail_seq=len(lens), max_q_len=max(lens), decode_tail_start=sum(lens), portion_lens=tuple(lens) if given else ())
        return MatrixLstmMixer._chunks(part, ctx, sum(lens))

    assert chunks([2000]) == 32 and chunks([200]) == 4 and chunks([200] * 8) == 32
    assert chunks([95]) == 0 and chunks([100] + [8] * 60) == 0 and chunks([1000] + [5] * 200) == 0
    assert chunks([2000], given=False) >= 32
    assert chunks([16384]) == 256 and chunks([20000]) == 0          # 256 chunks of 1.1 MB are allowed, 512 (the next size) are not
