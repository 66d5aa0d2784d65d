"""Attention over a compressed cache (latent attention).

Per token the layer keeps one latent vector ``c`` [kv_rank] (an RMS-normed projection of its input) and one rotated
key part ``k_r`` [rot_dim] that all heads share. Head a has the query ``[q_a | q_rot_a]`` ([dim | rot_dim], the
second part rotated by position), the key ``[W_uk_a c | k_r]`` and the value ``W_uv_a c``; scores are causal,
softmaxed, and the head's output may be gated by ``sigmoid(W_g h)_a`` before the output projection.

For single tokens the keys and values are never formed. With ``q~_a = W_uk_a^T q_a`` the score is ``(q~_a . c + q_rot_a . k_r) * scale``
and the output ``W_uv_a (sum_j p_j c_j)``: attention runs on the cached vectors themselves, with one key/value
"head" of width kv_rank + rot_dim for all query heads. Steps:

    one product     [W_q ; W_dkv ; W_g] h                          (``ops.linear``)
    latent_prepare  norm of the latent, rotations, cache write     (one kernel)
    head_gemm       q~ = W_uk^T q per head                         (one kernel)
    attention       over the latent pages                          (tensor cores in bfloat16 where rank and rot_dim
                                                                    are multiples of 16; the exact kernel otherwise
                                                                    and for the whole 32-bit path)
    head_gemm       W_uv per head, times the gate                  (one kernel)
    output product  W_o                                            (left to the residual stream)

That form costs heads * (2 kv_rank + rot_dim) multiply-adds a (query, key) pair, the plain one heads * (dim + rot_dim + value_dim),
3.4 times less at 128 + 64, 128 and a latent of 512, beside kv_rank * heads * (dim + value_dim) a key to expand it. So portions of prompts
in bfloat16 expand, where the head sizes are those of the tcgen05 kernel (``_expands`` says from how many keys on, ``__init__`` in which
models):

    one product, latent_prepare  as above
    latent_gather                the requests' latents out of their pages
    one product                  [W_uk ; W_uv] c: every head's keys and values (the experts' tcgen05 product, of one expert)
    latent_prefill_tc            attention over them, times the gate (tcgen05)
    output product               as above

Other forms, chosen by spec params: ``q_rank`` r > 0 sends the queries through a latent of their own,
``q = W_uq rms_norm(W_dq h)`` (tensors ``dq`` [r, hidden], ``dq.norm`` [r], ``uq`` in place of ``q``; the norm uses
``latent_eps``): W_dq joins the fused product, one kernel norms its columns and a second product makes the queries.
``sinks``: a tensor ``sink`` [heads]; exp(sink_a) joins the denominator of head a's softmax (no key, no value).
``output_gate`` ``full``: ``g`` is [heads * value_dim, hidden] and gates every output entry (the default form is one gate a
head). ``pairing`` ``halves``: rotated entry i turns with entry i + dims / 2 (the kernels turn neighbours (2i, 2i + 1)): the
rotated rows of the query and key projections are laid out pair by pair at load, which leaves every score as it is, and
``named_tensors`` gives the stored order back.

A layer with ``own_latent`` False has no W_dkv: its run is scheduled on another layer's cache slot without writing
it, and reads what that layer stored (latent after the norm, key part after the rotation).

Spec: ``num_heads``, ``head_dim`` (the unrotated query/key width), ``scale``, ``position`` (a rotary table; its
``head_dim`` is the number of rotated entries, pairs (2i, 2i+1)), params ``rot_dim``, ``value_dim``, ``kv_rank``,
``latent_eps``, ``own_latent``, ``output_gate``, ``q_rank``, ``sinks``, ``pairing``. Tensors under the prefix: ``q`` (or ``dq``,
``dq.norm``, ``uq``), ``dkv``, ``dkv.norm``, ``uk``, ``uv``, ``g``, ``sink``, ``o``.
"""

from __future__ import annotations

import torch

from ..csrc import ops
from .base import CacheRequest, Mixer, Projection, TensorDecl, build_part, register_part


class LatentAttention(Mixer):
    lazy_output = True
    # Portions go over expanded keys where one of their requests holds this many: the folded form walks a request's keys in one CTA, a
    # tile of 64 after the other at 2.3 us each, however few the tokens. Two such layers of 16 heads and nothing else, a step on the latents /
    # expanded, us: 2,000 tokens alone 911 / 586, 2,000 behind 8,000 3,644 / 1,034, 10 behind 30,000 2,937 / 1,831, 33 behind 2,000 512 / 498,
    # 1,000 alone 525 / 496, 512 alone 405 / 457, 100 behind 600 373 / 420. The line was drawn when the folded form ran on mma.sync (12 us a tile,
    # 2,000 alone 1,738); some 1,000 keys are where the forms are level now, and from 512 to there the latents would be 10 % faster. (The forms'
    # roundings are alike: their outputs differ by 0.0013 to 0.0015, the expanded form 1 % nearer to 64 bits.) Below it the folded form has
    # fewer launches. Many requests make the product that expands long while the walk stays what the longest one's is: at most
    # EXPAND_SHARE times the longest one's keys in all (on mma.sync 16 of 16 tokens behind 1,000 556 / 580).
    EXPAND_KEYS = 512
    EXPAND_SHARE = 8
    MAX_EXPANDED_BYTES = 1 << 28      # keys and values of a step, expanded, at most (the buffer, whose rows are a power of two)

    def __init__(self, spec, runtime):
        super().__init__(spec, runtime)
        s, p = spec, dict(spec.params)
        self.hidden, self.heads, self.dim = int(s.hidden), int(s.num_heads), int(s.head_dim)
        self.rot, self.vdim, self.rank = int(p["rot_dim"]), int(p["value_dim"]), int(p["kv_rank"])
        self.eps = float(p.get("latent_eps", 0.0))
        self.own_latent = bool(p.get("own_latent", True))
        self.gated = bool(p.get("output_gate", False))
        self.full_gate = p.get("output_gate") == "full"
        self.q_rank = int(p.get("q_rank", 0))
        self.has_sinks = bool(p.get("sinks", False))
        self.halves = p.get("pairing", "neighbours") == "halves"
        if p.get("pairing", "neighbours") not in ("neighbours", "halves") or self.q_rank < 0:
            raise ValueError("latent attention: `pairing` is neighbours or halves, `q_rank` not negative")
        self.scale = float(s.scale)
        if min(self.heads, self.dim, self.vdim, self.rank) <= 0 or self.rot <= 0:
            raise ValueError("latent attention needs positive heads, dim, rot_dim, value_dim and kv_rank")
        if self.rank > 512:
            raise ValueError(f"kv_rank {self.rank} is not supported by the latent attention kernel (up to 512 is)")
        self.position = build_part("position", s.position, runtime)
        self.rot_dims = int(s.position.head_dim)
        if self.rot_dims > self.rot or self.rot_dims % 2:
            raise ValueError(f"{self.rot_dims} rotated entries do not fit a rotated part of {self.rot}")
        self.q_dim = self.heads * (self.dim + self.rot)
        self.q_cols = self.q_rank if self.q_rank else self.q_dim        # what the fused product makes of the queries
        self.kv_dim = self.rank + self.rot if self.own_latent else 0
        self.g_dim = (self.heads * self.vdim if self.full_gate else self.heads) if self.gated else 0
        # columns of the fused product, each block starting at a multiple of 8 so that rows of 16-bit numbers stay
        # 16-byte aligned inside it
        self.q_off = 0
        self.kv_off = -(-self.q_cols // 8) * 8
        self.g_off = self.kv_off + -(-self.kv_dim // 8) * 8
        self.proj_dim = -(-(self.g_off + self.g_dim) // 8) * 8
        self.w_in = self.w_ukv = self.w_uk = self.w_uv = self.w_o = self.latent_w = self.w_uq = self.q_norm_w = self.sinks = None
        # rotated entries in the order the kernels pair them: new entry 2i is old entry i, new entry 2i + 1 old entry i + dims / 2
        half = self.rot_dims // 2
        order = [j for i in range(half) for j in (i, i + half)] + list(range(self.rot_dims, self.rot))
        self.rot_order = torch.tensor(order, dtype=torch.long) if self.halves else None
        # In a model with a matrix LSTM the layer stays on the latents in prompts too. Both forms are as far from 64 bits (layers alone:
        # 0.0018 of the result each, expanded a hundredth closer), but the matrix LSTM divides by a sum that can vanish: what the other
        # rounding changed in front of it then grew to 0.03 to 0.06 of the logits in 4 of 24 passes of the Netusun shape, more than
        # two runs of this path may differ by.
        self._expand = "mlstm" not in runtime.mixer_kinds and ops.latent_prefill_supported(runtime.dtype, self.dim, self.vdim, self.rot, self.rank)
        self.sizes_by_context = self._expand
        self._fast = ops.latent_tc_supported(runtime.dtype, self.heads, self.rank, self.rot)

    # ----------------------------------------------------------------- weights
    def _n(self, short):
        return self.spec.prefix + short

    def declare(self):
        d = {self._n("uk"): TensorDecl((self.heads * self.dim, self.rank)),
             self._n("uv"): TensorDecl((self.heads * self.vdim, self.rank)), self._n("o"): TensorDecl((self.hidden, self.heads * self.vdim))}
        if self.q_rank:
            d[self._n("dq")] = TensorDecl((self.q_rank, self.hidden))
            d[self._n("dq.norm")] = TensorDecl((self.q_rank,), "vector")
            d[self._n("uq")] = TensorDecl((self.q_dim, self.q_rank))
        else:
            d[self._n("q")] = TensorDecl((self.q_dim, self.hidden))
        if self.own_latent:
            d[self._n("dkv")] = TensorDecl((self.rank + self.rot, self.hidden))
            d[self._n("dkv.norm")] = TensorDecl((self.rank,), "vector")
        if self.gated:
            d[self._n("g")] = TensorDecl((self.g_dim, self.hidden))
        if self.has_sinks:
            d[self._n("sink")] = TensorDecl((self.heads,), "vector")
        d.update(self.position.declare())
        return d

    def _pair_rows(self, t, first: int, blocks: int, stride: int, inverse: bool = False):
        """Rows ``first + b * stride .. + rot`` of ``t`` for b < blocks (the rotated parts) in the kernels' order of pairs."""
        if self.rot_order is None:
            return t
        order = torch.argsort(self.rot_order) if inverse else self.rot_order
        t = t.clone()
        for b in range(blocks):
            at = first + b * stride
            t[at:at + self.rot] = t[at:at + self.rot].index_select(0, order.to(t.device))
        return t

    def bind(self, weights):
        q = self._pair_rows(weights[self._n("uq" if self.q_rank else "q")], self.dim, self.heads, self.dim + self.rot)
        w = torch.zeros((self.proj_dim, self.hidden), dtype=q.dtype, device=q.device)
        if self.q_rank:
            w[:self.q_rank] = weights[self._n("dq")]
            self.w_uq, self.q_norm_w = q.contiguous(), weights[self._n("dq.norm")]
        else:
            w[:self.q_dim] = q
        if self.own_latent:
            w[self.kv_off:self.kv_off + self.kv_dim] = self._pair_rows(weights[self._n("dkv")], self.rank, 1, 0)
            self.latent_w = weights[self._n("dkv.norm")]
        if self.gated:
            w[self.g_off:self.g_off + self.g_dim] = weights[self._n("g")]
        if self.has_sinks:
            self.sinks = weights[self._n("sink")]
        self.w_in = w
        # W_uk's rows, then W_uv's, so that one product expands both
        self.w_ukv = torch.cat([weights[self._n("uk")], weights[self._n("uv")]]).contiguous()
        self.w_uk, self.w_uv = self.w_ukv[:self.heads * self.dim], self.w_ukv[self.heads * self.dim:]
        self.w_o = weights[self._n("o")]
        self.position.bind(weights)

    def named_tensors(self):
        out = {self._n("uk"): self.w_uk, self._n("uv"): self.w_uv, self._n("o"): self.w_o}
        if self.q_rank:
            out[self._n("dq")], out[self._n("dq.norm")] = self.w_in[:self.q_rank], self.q_norm_w
            out[self._n("uq")] = self._pair_rows(self.w_uq, self.dim, self.heads, self.dim + self.rot, inverse=True)
        else:
            out[self._n("q")] = self._pair_rows(self.w_in[:self.q_dim], self.dim, self.heads, self.dim + self.rot, inverse=True)
        if self.own_latent:
            out[self._n("dkv")] = self._pair_rows(self.w_in[self.kv_off:self.kv_off + self.kv_dim], self.rank, 1, 0, inverse=True)
            out[self._n("dkv.norm")] = self.latent_w
        if self.gated:
            out[self._n("g")] = self.w_in[self.g_off:self.g_off + self.g_dim]
        if self.has_sinks:
            out[self._n("sink")] = self.sinks
        out.update(self.position.named_tensors())
        return out

    # ------------------------------------------------------------------- cache
    def cache_request(self):
        return CacheRequest(tensors=(("latent", 1, self.rank), ("key_rot", 1, self.rot)))

    # ----------------------------------------------------------------- forward
    def forward(self, x, ctx, cache, lazy_output: bool = False):
        tokens = x.shape[0]
        if self.own_latent != bool(cache.writes):
            raise ValueError("a latent attention layer writes the cache exactly when it has a latent projection of its own")
        proj = self.rt.buffer("latent_proj", tokens, self.proj_dim)
        ops.linear(x, self.w_in, proj)
        width = self.rank + self.rot
        qa = self.rt.buffer("latent_q", tokens, self.heads * width)
        latent, key_rot = cache.tensors["latent"], cache.tensors["key_rot"]
        cos, sin = self.position.tables()
        seq, pos = ctx.seq_of_token[:tokens], ctx.positions[:tokens]
        q, q_ld, q_off = proj, self.proj_dim, self.q_off
        if self.q_rank:         # queries through their own latent: norm of its columns, then the second product
            q_latent = self.rt.buffer("latent_q_latent", tokens, self.q_rank)
            ops.rms_norm_cols(proj, 0, self.q_rank, self.q_norm_w, q_latent, self.eps)
            q, q_ld, q_off = self.rt.buffer("latent_q_full", tokens, self.q_dim), self.q_dim, 0
            ops.linear(q_latent, self.w_uq, q)
        ops.latent_prepare(proj, self.q_off, self.kv_off if self.own_latent else -1, qa, pos, seq,
                           ctx.slot_mapping[cache.group][:tokens] if cache.writes else None, cos, sin, self.latent_w, self.eps,
                           latent, key_rot, self.heads, self.dim, self.rot, self.rot_dims, self.rank, q=q if self.q_rank else None)
        attn = self.rt.buffer("latent_out", tokens, self.heads * self.vdim)
        first = 0               # rows from here on go over the latents themselves
        if self._expands(ctx, tokens):
            first = min(ctx.decode_tail_start, tokens)
            self._attend_expanded(q, q_off, qa, attn[:first], latent, key_rot, proj, ctx, cache)
        if tokens > first:
            mixed, gate, rows = self.rt.buffer("latent_mixed", tokens, self.heads * self.rank), proj if self.gated else None, slice(first, tokens)
            q_in, q_out, o_in, o_out = (q, qa, mixed, attn) if not first else (q[rows], qa[rows], mixed[rows], attn[rows])
            # q~[t, a, :] = q[t, a, :dim] @ W_uk[a]          W_uk [heads * dim, rank]: B_a[k, n] = W_uk[a * dim + k, n]
            ops.head_gemm(q_in, q_ld, self.dim + self.rot, self.w_uk, self.dim * self.rank, self.rank, 1, q_out, self.heads * width, width,
                          tokens - first, self.heads, self.rank, self.dim, a_off=q_off)
            self._attend(qa, mixed, latent, key_rot, ctx, cache, tokens, first)
            # o[t, a, :] = W_uv[a] mixed[t, a, :]            W_uv [heads * vdim, rank]: B_a[k, n] = W_uv[a * vdim + n, k]
            ops.head_gemm(o_in, self.heads * self.rank, self.rank, self.w_uv, self.vdim * self.rank, 1, self.rank, o_out, self.heads * self.vdim,
                          self.vdim, tokens - first, self.heads, self.vdim, self.rank, gate=gate if gate is None or not first else gate[rows],
                          ldg=self.proj_dim, gate_off=self.g_off, gate_per_output=self.full_gate)
        if lazy_output:
            return Projection(attn, self.w_o)
        out = self.rt.buffer("mixer_out", tokens, self.hidden)
        ops.linear(attn, self.w_o, out)
        return out

    def _expanded_rows(self, keys) -> int:
        return max(2048, 1 << (keys - 1).bit_length())          # few sizes, for the scratch and for the copies' descriptors

    def _expands(self, ctx, tokens) -> bool:
        """Whether this step's portions go over expanded keys and values."""
        keys, longest = ctx.portion_keys, ctx.portion_longest
        return (self._expand and ctx.decode_tail_start > 0 and longest >= self.EXPAND_KEYS and keys <= self.EXPAND_SHARE * longest
                and self._expanded_rows(keys) * self.heads * 2 * (self.dim + self.vdim) <= self.MAX_EXPANDED_BYTES)

    def _attend_expanded(self, q, q_off, qa, out, latent, key_rot, proj, ctx, cache):
        keys, seqs = ctx.portion_keys, ctx.decode_tail_seq
        rows = self._expanded_rows(keys)
        c = self.rt.scratch("latent_dense", rows * self.rank, self.rt.dtype)[:rows * self.rank].view(rows, self.rank)
        k_rot = self.rt.scratch("latent_dense_rot", rows * self.rot, self.rt.dtype)[:rows * self.rot].view(rows, self.rot)
        kv_dim = self.heads * (self.dim + self.vdim)
        kv = self.rt.scratch("latent_expanded", rows * kv_dim, self.rt.dtype)[:rows * kv_dim].view(rows, kv_dim)
        filled = self.rt.scratch("latent_filled", 2, torch.int32)
        ops.latent_gather(latent, key_rot, ctx.block_table[cache.group], ctx.ctx_len, seqs, cache.page_size, c[:keys], k_rot[:keys], filled)
        # the experts' product with one expert, whose rows are those that were filled
        if not ops.grouped_gemm_tc(c, self.w_ukv.view(1, kv_dim, self.rank), filled, kv, rows):
            raise ops.KernelError("the product that expands keys and values does not take the sizes")
        ops.latent_prefill_tc(q, q_off, qa, self.rank, self.rank + self.rot, kv, k_rot, out, ctx.q_start, ctx.q_len, ctx.ctx_len, seqs,
                              self.heads, self.scale, sinks=self.sinks, gate=proj if self.gated else None, gate_off=self.g_off,
                              gate_per_output=self.full_gate, kv_head_stride=self.dim, kv_v_off=self.heads * self.dim)

    def _attend(self, qa, mixed, latent, key_rot, ctx, cache, tokens, first: int = 0):
        """Attention over the latents themselves for the rows from ``first`` on (0, or where the decode tail starts)."""
        table = ctx.block_table[cache.group]
        if not self._fast:
            # the exact kernel: the whole 32-bit path, and sizes the tensor-core kernel refuses
            ops.latent_attention(qa[first:], mixed[first:], latent, key_rot, table, ctx.seq_of_token[first:tokens], ctx.positions[first:tokens],
                                 self.heads, self.rank, self.rot, cache.page_size, self.scale, sinks=self.sinks)
            return
        geometry = (self.heads, self.rank, self.rot, cache.page_size, self.scale)
        split = min(ctx.decode_tail_start, tokens)          # portions before, single tokens after
        if split > first and not ops.latent_attention_tc5(qa, mixed, latent, key_rot, table, ctx.q_start, ctx.q_len, ctx.ctx_len, ctx.decode_tail_seq,
                                                          max(ctx.max_q_len, 2), *geometry, sinks=self.sinks):
            ops.latent_attention_tc(qa, mixed, None, latent, key_rot, table, ctx.q_start, ctx.q_len, ctx.ctx_len, ctx.seq_of_token, 0,
                                    ctx.decode_tail_seq, 0, split, max(ctx.max_q_len, 2), *geometry, sinks=self.sinks)
        if tokens > split:
            n = tokens - split
            # enough CTAs to fill the device, down to one tile of keys a split: a tile of 64 keys takes a CTA some 12 us, one after the other
            tiles = n * -(-self.heads // 16)
            splits = max(1, min(-(-ctx.context_bound // 64), -(-296 // tiles), 64))
            per_split = -(-(-(-ctx.context_bound // splits)) // 64) * 64
            splits = max(1, -(-ctx.context_bound // per_split))
            partial = None
            if splits > 1:
                partial = self.rt.scratch("latent_splits", tokens * self.heads * splits * (self.rank + 2))
            ops.latent_attention_tc(qa, mixed, partial, latent, key_rot, table, ctx.q_start, ctx.q_len, ctx.ctx_len, ctx.seq_of_token,
                                    ctx.decode_tail_seq, n, split, n, 1, *geometry, splits=splits, keys_per_split=per_split, sinks=self.sinks)


register_part("mixer", "latent_attention", LatentAttention)
