"""Latent attention whose portions go over expanded keys and values, as a model and the engine drive it: whole prompts, portions
beside single tokens, the byte limit, full portions replayed from captured graphs at positions far past the captured one, and a
latent layer inside a parallel mixer. Against the plain float64 implementation (``plain_nidilix``)."""

import dataclasses

import pytest
import torch

import nidilix_cases as cases
import plain_nidilix as plain
from helpers import compare_logits, seeded_tokens, write_model_dir

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def two_layers(rank):
    """The head sizes of the tcgen05 kernel; the second layer borrows the first one's latents."""
    heads = cases.attention(3, 128, 64, 64, 128, rank)
    return cases.config(96, 131, [(heads, None), (cases.attention(3, 128, 64, 64, 128, rank, kv_from=0), None)], mult=0.5)


class Case:
    def __init__(self, tmp_models, rank, seed=41):
        self.cfg = two_layers(rank)
        state = cases.seeded_state(self.cfg, seed)
        self.folder = write_model_dir(str(tmp_models / f"latent_expanded_{rank}"), self.cfg, state, torch.bfloat16)
        self.state = {k: v.bfloat16() for k, v in state.items()}
        self.want = {}

    def logits(self, tokens):
        key = tuple(tokens)
        if key not in self.want:
            self.want[key] = plain.forward(self.cfg, self.state, list(tokens))
        return self.want[key]


@pytest.fixture(scope="module")
def models(tmp_models):
    return {rank: Case(tmp_models, rank) for rank in (48, 40)}       # 40: the tensor-core kernel over the latents refuses it


@pytest.fixture
def expansions(monkeypatch):
    """The expanded kernel's calls, the rows of each; requests of 64 keys and more are worth expanding."""
    from stride_b200.csrc import ops
    from stride_b200.parts.latent_attention import LatentAttention
    monkeypatch.setattr(LatentAttention, "EXPAND_KEYS", 64)
    calls, run = [], ops.latent_prefill_tc
    monkeypatch.setattr(ops, "latent_prefill_tc", lambda *a, **k: (calls.append(a[7].shape[0]), run(*a, **k))[1])
    return calls


def engine_for(case, **options):
    from stride_b200 import Engine
    options = {"block_size": 16, "num_blocks": 80, "max_batch_tokens": 256, "max_batch_seqs": 6, "max_model_len": 400, **options}
    return Engine(case.folder, dtype="bfloat16", **options)


def check(got, case, tokens, rows, label):
    ok, msg = compare_logits(got.cpu(), case.logits(tokens)[rows], "bfloat16")
    assert ok, f"{label}: {msg}"


def open_request(engine, key, n):
    engine.cache.open(key, "u")
    assert engine.cache.ensure(key, n, 0)


def full_portions(engine, case, key, tokens, size):
    """A prompt in portions that fill the token budget; logits of the last row of each."""
    open_request(engine, key, len(tokens))
    for at in range(0, len(tokens), size):
        want = [size - 1] if at + size >= len(tokens) or at % (2 * size) else []
        got = engine.forward([(key, tokens[at:at + size], at, want)])
        if want:
            check(got, case, tokens, [at + size - 1], f"request {key}, portion at {at}")
    engine.cache.close(key)


@pytest.mark.parametrize("bucketed", [True, False])
def test_full_portions_replayed_from_graphs(gpu, models, expansions, monkeypatch, bucketed):
    """Four portions of 64 tokens, with a context bucket that ends behind each of them; then another prompt over the same graphs.
    A model that gives no bound for its captured portions (a layer without ``parts``, say) stays on the latents: a graph captured at
    the first portion must not go on to expand that portion's keys alone."""
    from stride_b200.engine.runner import ModelRunner
    from stride_b200.parts.model import DecoderModel
    monkeypatch.setattr(ModelRunner, "CONTEXT_BUCKET_BASE", 64)
    if not bucketed:
        monkeypatch.setattr(DecoderModel, "sizes_by_context", False)
    case = models[48]
    engine = engine_for(case, max_batch_tokens=64)
    for key in (1, 2):
        full_portions(engine, case, key, seeded_tokens(256, case.cfg["vocab"], 900 + key), 64)
    bounds = {k[2:] for k in engine.runner._graphs if k[0] == "portion"}
    assert (len(bounds) >= 3 and len(expansions) > 0) if bucketed else (bounds == {()} and not expansions)
    assert engine.runner.graph_replays == 8


def register_parallel():
    from stride_b200.config import MixerSpec, register_architecture
    from stride_b200.config.nidilix import NidilixConfig

    class InParallel:
        """The Nidilix design with every mixer as the one branch of a parallel mixer."""

        def __init__(self, d):
            self.d = dict(d)

        @classmethod
        def from_dict(cls, d):
            return cls(d)

        def to_dict(self):
            return dict(self.d)

        def to_model_spec(self):
            spec = NidilixConfig.from_dict(dict(self.d, architecture="Nidilix")).to_model_spec()
            layers = tuple(dataclasses.replace(l, mixer=MixerSpec("parallel", hidden=spec.hidden, prefix=l.mixer.prefix,
                                                                  params=(("branches", ((l.mixer, 1.0),)),))) for l in spec.layers)
            return dataclasses.replace(spec, layers=layers)

    register_architecture("ToyLatentInParallel", InParallel)


def test_a_latent_branch_of_a_parallel_mixer_in_full_portions(gpu, models, expansions, monkeypatch, tmp_models):
    from stride_b200.engine.runner import ModelRunner
    register_parallel()
    monkeypatch.setattr(ModelRunner, "CONTEXT_BUCKET_BASE", 64)
    cfg = dict(two_layers(48), architecture="ToyLatentInParallel")
    cfg["layers"] = cfg["layers"][:1]
    case = Case.__new__(Case)
    case.cfg, case.want = dict(cfg, architecture="Nidilix"), {}
    state = cases.seeded_state(case.cfg, 43)
    case.folder = write_model_dir(str(tmp_models / "latent_in_parallel"), cfg, state, torch.bfloat16)
    case.state = {k: v.bfloat16() for k, v in state.items()}
    engine = engine_for(case, max_batch_tokens=64)
    assert engine.model.sizes_by_context
    full_portions(engine, case, 1, seeded_tokens(256, cfg["vocab"], 911), 64)
    assert expansions and engine.runner.graph_replays == 4


@pytest.mark.parametrize("rank", [48, 40])
def test_portions_beside_single_tokens(gpu, models, expansions, monkeypatch, rank):
    """A whole prompt; then a portion behind it and another request's first one beside two single tokens, which go over the latents:
    through the tensor-core kernel, or (a rank it refuses) the exact one, which is given their rows alone."""
    from stride_b200.csrc import ops
    from stride_b200.parts.latent_attention import LatentAttention
    monkeypatch.setattr(LatentAttention, "EXPAND_KEYS", 1)
    exact, run = [], ops.latent_attention
    monkeypatch.setattr(ops, "latent_attention", lambda *a, **k: (exact.append(a[0].shape[0]), run(*a, **k))[1])
    case, vocab = models[rank], models[rank].cfg["vocab"]
    engine = engine_for(case)
    tokens = {key: seeded_tokens(n, vocab, 700 + key) for key, n in ((1, 150), (2, 90), (3, 40), (4, 70))}
    for key, t in tokens.items():
        open_request(engine, key, len(t))
    check(engine.forward([(1, tokens[1][:120], 0, list(range(120)))]), case, tokens[1], list(range(120)), "whole prompt")
    assert expansions == [120, 120]             # two layers
    engine.forward([(2, tokens[2][:89], 0, []), (3, tokens[3][:39], 0, [])])
    exact.clear()
    got = engine.forward([(1, tokens[1][120:], 120, list(range(30))), (4, tokens[4], 0, list(range(70))), (2, tokens[2][89:], 89, [0]),
                          (3, tokens[3][39:], 39, [0])])
    assert expansions[-1] == 100 and exact == ([2, 2] if rank == 40 else [])
    for key, rows, at in ((1, range(120, 150), 0), (4, range(70), 30), (2, [89], 100), (3, [39], 101)):
        check(got[at:at + len(rows)], case, tokens[key], list(rows), f"request {key} of the mixed step")


def test_the_rule_and_the_byte_limit(gpu, models, expansions, monkeypatch):
    """Short requests, too many keys beside the longest one's, and a buffer past the limit stay on the latents."""
    from stride_b200.parts.latent_attention import LatentAttention
    case = models[48]
    tokens = {key: seeded_tokens(n, case.cfg["vocab"], 720 + key) for key, n in ((1, 80), (2, 30), (3, 30))}

    def run(expanded, keys=80, share=8, limit=1 << 28):
        for name, value in (("EXPAND_KEYS", keys), ("EXPAND_SHARE", share), ("MAX_EXPANDED_BYTES", limit)):
            monkeypatch.setattr(LatentAttention, name, value)
        engine = engine_for(case)
        for key, t in tokens.items():
            open_request(engine, key, len(t))
        before = len(expansions)
        got = engine.forward([(key, t, 0, list(range(len(t)))) for key, t in tokens.items()])
        at = 0
        for key, t in tokens.items():
            check(got[at:at + len(t)], case, t, list(range(len(t))), f"request {key}")
            at += len(t)
        assert (len(expansions) > before) == expanded

    run(True)
    run(False, keys=81)
    run(False, share=1)
    # 140 keys take a buffer of 2,048 rows of 3 heads of 256 numbers
    run(True, limit=2048 * 3 * 512)
    run(False, limit=2048 * 3 * 512 - 1)


def test_weights_are_handed_out_as_they_are_held(gpu, models):
    """A change to what ``get_weight`` gives is a change to the model, also of the two matrices that one product expands with."""
    case = models[48]
    engine = engine_for(case)
    tokens = seeded_tokens(20, case.cfg["vocab"], 731)
    open_request(engine, 1, 20)
    before = engine.forward([(1, tokens, 0, [19])]).clone()
    for name in ("l0.mix.uk", "l0.mix.uv"):
        weight = engine.get_weight(name)
        assert weight.shape == case.state[name].shape and torch.equal(weight.cpu(), case.state[name])
        weight.zero_()
        assert not bool(engine.get_weight(name).any())
        after = engine.forward([(1, tokens, 0, [19])]).clone()
        assert not torch.equal(before, after)
        before = after


@pytest.mark.parametrize("lstm", [False, True])
def test_query_latents_expand_unless_the_model_holds_a_matrix_lstm(gpu, expansions, monkeypatch, tmp_models, lstm):
    import netusun_cases
    import plain_netusun
    from stride_b200.parts.latent_attention import LatentAttention
    monkeypatch.setattr(LatentAttention, "EXPAND_KEYS", 1)
    layers = [(netusun_cases.latent(3, 128, 64, 128, 48, 32), netusun_cases.dense(72))]
    if lstm:
        layers.append((netusun_cases.lstm(2, 24, 16), None))
    cfg = netusun_cases.config(96, 131, layers)
    state = netusun_cases.seeded_state(cfg, 47)
    folder = write_model_dir(str(tmp_models / f"latent_netusun_{lstm}"), cfg, state, torch.bfloat16)
    case = Case.__new__(Case)
    case.folder = folder
    engine = engine_for(case)
    tokens = seeded_tokens(140, 131, 733)
    open_request(engine, 1, 140)
    got = engine.forward([(1, tokens, 0, list(range(0, 140, 7)))]).cpu()
    assert bool(expansions) == (not lstm)
    if not lstm:
        want = plain_netusun.forward(cfg, {k: v.bfloat16().double() for k, v in state.items()}, tokens)[list(range(0, 140, 7))]
        error = float((got.double() - want).norm() / want.norm())
        assert error <= 0.03, error         # bfloat16 through one layer; a lost key or rotation changes rows outright


@pytest.mark.parametrize("lens,rows", [([5, 0, 17], 40), ([64], 64), ([100, 200], 150)])
def test_the_gather_says_how_many_rows_it_filled(gpu, lens, rows):
    """What the product that expands them is bounded by; never more than the rows there are."""
    from stride_b200.csrc import ops
    page, rank, rot = 16, 48, 64
    pages = [-(-n // page) for n in lens]
    table = torch.full((len(lens), max(pages)), -1, dtype=torch.int32)
    for s, n in enumerate(pages):
        table[s, :n] = torch.arange(n) + sum(pages[:s])
    latent, key_rot = (torch.randn(sum(pages), 1, page, n, device="cuda").bfloat16() for n in (rank, rot))
    c, k_rot = (torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda") for n in (rank, rot))
    filled = torch.full((3,), -5, dtype=torch.int32, device="cuda")
    ops.latent_gather(latent, key_rot, table.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), len(lens), page, c, k_rot, filled[:2])
    total = min(sum(lens), rows)
    assert filled.tolist() == [0, total, -5]
    assert bool((c[total:] == 7.0).all()) and not bool((c[:total] == 7.0).all(1).any())
