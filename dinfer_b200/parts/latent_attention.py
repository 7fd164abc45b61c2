"""Attention over a cached latent (multi-head latent attention), run in its absorbed form.

The design: queries go through a latent (``cq = RMSNorm(W_dq x)``, ``q = W_uq cq``, per head ``D`` unrotated and
``P`` rotated elements); keys and values come from one latent per token, ``c = RMSNorm((W_dkv x)[:R])``, plus one
rotated key part ``kr = rot((W_dkv x)[R:])`` shared by all heads: ``k_h = [W_uk[h] c | kr]``, ``v_h = W_uv[h] c``.
Only ``[c | kr]`` is cached (one row of R + P per token, pages ``[pages, 1, 1, page, R + P]``).

Absorbed: ``q_h . k_h = (W_uk[h]^T q_h[:D]) . c + q_h[D:] . kr`` and ``sum_j p_j v_hj = W_uv[h] (sum_j p_j c_j)``, so a
step never expands a cached row into per-head keys and values:

  [cq | c | kr] = x [W_dq; W_dkv]^T        one stacked product
  norm(cq), norm(c), rot(kr) -> cache      one kernel
  q = cq W_uq^T
  q_lat[:, h] = [ q[:, h, :D] W_uk[h] | rot(q[:, h, D:]) ]      batched product + one kernel
  o_lat[:, h] = softmax(q_lat[:, h] . rows * scale) rows[:, :R] multi-query attention over the latent cache
  o[:, h] = o_lat[:, h] W_uv[h]^T          batched product
  y = o W_o^T

Portions of several tokens are worth expanding the rows they see (``LatentAttention._expanded``): from q on

  rows = the cached rows of the portions' requests, gathered;  kv = c [W_uk; W_uv]^T    one product for all heads
  o[:, h] = softmax((q_h . [k_h | kr]) * scale) v_h

A layer with ``own_kv`` False has no W_dkv: its schedule entry reads another entry's cache (``cache.write`` False)
with its own W_uk, W_uv and queries.
"""
from __future__ import annotations

from typing import Dict, List, Optional

import torch

from ..kernels import latent_ops, ops
from ..kernels.lib import add_launches, num_sms
from .base import MIXERS, POSITION_ENCODINGS, BuildEnv, CacheBinding, KvCacheNeed, Mixer, StepContext, build_part
from .linear import Linear
from .spec import PartSpec, TensorDecl


@MIXERS.register("latent_attention")
class LatentAttention(Mixer):
    """params: ``num_heads``, ``nope_dim`` (D), ``rope_dim`` (P), ``v_dim``, ``kv_rank`` (R), ``q_rank``, ``scale``,
    ``eps`` (of the two latent norms), ``position`` (a PartSpec of a table rotation over the ``rope_dim`` part),
    ``own_kv`` (False: no down projection for keys and values, the entry reads another entry's cache), optional
    ``window``, ``cache_block_size``, ``sink`` (tensor name of one number per head: the softmax of head h has one more
    term ``exp(sink_h)`` that carries no value and is not scaled), ``gate_proj`` (tensor name of ``W_g`` [H * v_dim,
    width]: the heads' outputs are multiplied by ``sigmoid(W_g x)`` before the output projection; it rides in the
    stacked down projection), ``out_float32``, and the tensor names ``q_down``, ``q_norm``, ``q_up``, ``kv_down``, ``kv_norm``,
    ``k_up``, ``v_up``, ``o_proj``."""

    def __init__(self, params, env: BuildEnv, prefix=""):
        super().__init__(params, env, prefix)
        p = self.params
        self.hidden = env.hidden_size
        self.H, self.D, self.P = int(p["num_heads"]), int(p["nope_dim"]), int(p["rope_dim"])
        self.V, self.R, self.Rq = int(p["v_dim"]), int(p["kv_rank"]), int(p["q_rank"])
        self.scale = float(p["scale"]) if p.get("scale") is not None else 1.0 / float(self.D + self.P) ** 0.5
        self.eps = float(p.get("eps", 1e-6))
        self.own_kv = bool(p.get("own_kv", True))
        self.window = p.get("window")
        self.page_size = p.get("cache_block_size")
        pos: PartSpec = p.get("position") or PartSpec("none")
        self.position = build_part(POSITION_ENCODINGS, pos, env, prefix)
        if not self.position.fused:
            raise ValueError("latent attention rotates by a table (a position encoding its kernels apply)")
        # pairs (2i, 2i + 1), or (i, i + rot / 2) for a table rotation of the other style
        self.halves = self.position.fused_table() is not None and not getattr(self.position, "interleaved", False)
        self.sink_name = prefix + p["sink"] if p.get("sink") else None
        self.gate_name = prefix + p["gate_proj"] if p.get("gate_proj") else None
        self.out_float32 = bool(p.get("out_float32", False))
        self.sinks = None
        n = lambda key, default: prefix + p.get(key, default)
        self.names = {"dq": n("q_down", "q_down.weight"), "qn": n("q_norm", "q_norm.weight"), "uq": n("q_up", "q_up.weight"),
                      "dkv": n("kv_down", "kv_down.weight"), "kvn": n("kv_norm", "kv_norm.weight"),
                      "uk": n("k_up", "k_up.weight"), "uv": n("v_up", "v_up.weight"), "o": n("o_proj", "o_proj.weight")}
        self.down: Optional[Linear] = None
        self.uq: Optional[Linear] = None
        self.o: Optional[Linear] = None
        self.q_norm_w = self.kv_norm_w = self.uk_t = self.uv = None

    def declare(self) -> List[TensorDecl]:
        H, D, P, V, R, Rq, h = self.H, self.D, self.P, self.V, self.R, self.Rq, self.hidden
        d = [TensorDecl(self.names["dq"], (Rq, h)), TensorDecl(self.names["qn"], (Rq,), init="ones"),
             TensorDecl(self.names["uq"], (H * (D + P), Rq)), TensorDecl(self.names["uk"], (H * D, R)),
             TensorDecl(self.names["uv"], (H * V, R)), TensorDecl(self.names["o"], (h, H * V))]
        if self.own_kv:
            d += [TensorDecl(self.names["dkv"], (R + P, h)), TensorDecl(self.names["kvn"], (R,), init="ones")]
        if self.sink_name:
            d.append(TensorDecl(self.sink_name, (H,)))
        if self.gate_name:
            d.append(TensorDecl(self.gate_name, (H * V, h)))
        return d

    def bind(self, tensors: Dict[str, torch.Tensor]) -> None:
        t = {k: tensors[v] for k, v in self.names.items() if v in tensors}
        rows = [t["dq"]] + ([t["dkv"]] if self.own_kv else [])
        # the gate's rows ride behind the latents, from a multiple of 8 columns on (zero rows between)
        self.low_width = sum(x.shape[0] for x in rows)
        self.gate_at = (self.low_width + 7) // 8 * 8
        if self.gate_name:
            g = tensors[self.gate_name]
            if self.gate_at > self.low_width:
                rows.append(g.new_zeros((self.gate_at - self.low_width, g.shape[1])))
            rows.append(g)
        dt = torch.float32 if any(x.dtype == torch.float32 for x in rows) else rows[0].dtype
        self.down = Linear(torch.cat([x.to(dt) for x in rows], dim=0))           # [Rq (+ R + P) (+ H V), h], stacked once
        if self.sink_name:
            self.sinks = tensors[self.sink_name].float().contiguous()
        self.uq = Linear(t["uq"])
        self.o = Linear(t["o"])
        self.q_norm_w = t["qn"].contiguous()
        if self.own_kv:
            self.kv_norm_w = t["kvn"].to(self.q_norm_w.dtype).contiguous()
        # per head: W_uk[h] is [D, R]; the absorbing product wants it as [R, D] (out, in)
        self.uk_t = t["uk"].reshape(self.H, self.D, self.R).transpose(1, 2).contiguous()
        self.uv = t["uv"].reshape(self.H, self.V, self.R).contiguous()
        # [H (D + V), R]: what makes a row's keys and values of all heads, head after head
        self.ukv = None
        if latent_ops.expanded_supported(t["uk"].dtype, self.R, self.P, self.D, self.V) and t["uv"].dtype == t["uk"].dtype:
            self.ukv = Linear(torch.cat([t["uk"].reshape(self.H, self.D, self.R), self.uv], dim=1).reshape(-1, self.R))

    def cache_need(self):
        return KvCacheNeed(1, self.R + self.P, self.window, int(self.page_size) if self.page_size else None, planes=1)

    def kernel_libraries(self):
        expanded = ["latent_expanded"] + self.ukv.kernel_libraries() if self.ukv is not None and self.env.act_dtype == torch.bfloat16 else []
        return (["latent_post", "attention_latent", "gemm_f32"] + expanded + (["elementwise"] if self.gate_name else []) + self.down.kernel_libraries() + self.uq.kernel_libraries()
                + self.o.kernel_libraries())

    def forward(self, x, ctx: StepContext, cache: CacheBinding, sink=None):
        H, D, P, V, R, Rq = self.H, self.D, self.P, self.V, self.R, self.Rq
        g = ctx.groups[cache.group]
        T = x.shape[0]
        table = self.position.fused_table()
        full = self.down(x)                                              # [T, Rq (+ R + P) (+ gate)]
        low = full[:, :self.low_width]
        write = self.own_kv and cache.write
        if self.own_kv and not write:
            raise RuntimeError("a latent attention layer with its own down projection must own its cache entry")
        latent_ops.latent_down_post(low, ctx.positions, self.q_norm_w, Rq, self.kv_norm_w if write else None, R, P,
                                    self.eps, table, cache.kv if write else None, g.slot_mapping if write else None,
                                    halves=self.halves)
        q = self.uq(low[:, :Rq])                                         # [T, H (D + P)]
        expanded = self._expanded(ctx, q.dtype)
        # (a dummy portion of one token in a captured graph belongs to neither way: its row has to hold something finite)
        make = torch.zeros if expanded is not None and ctx.decode_splits else torch.empty
        o = make((T, H, V), dtype=q.dtype, device=q.device)
        if expanded is None or ctx.any_decode:
            # head-major storage, seen as [T, H, *]: the batched products then write whole matrices per head
            q_lat = torch.empty((H, T, R + P), dtype=q.dtype, device=q.device).transpose(0, 1)
            o_lat = torch.empty((H, T, R), dtype=q.dtype, device=q.device).transpose(0, 1)
            rows = (q, ctx.positions, q_lat, o_lat, o)
            if expanded is not None:                         # the rows from the first single token to the last
                a, z = self._single_rows(ctx)
                rows = tuple(t[a:z] for t in rows)
            q_, positions, q_lat_, o_lat_, o_ = rows
            self.absorb(q_.view(-1, H, D + P)[:, :, :D], self.uk_t, q_lat_[:, :, :R])
            latent_ops.latent_q_rope(q_, positions, table, q_lat_, H, D, P, R, halves=self.halves)
            self.attend(q_lat, o_lat, cache.kv, g, ctx, singles=expanded is not None)
            self.absorb(o_lat_, self.uv, o_)
        if expanded is not None:
            self.attend_expanded(q, o, cache.kv, g, ctx, table, *expanded)
        o = o.view(T, H * V)
        if self.gate_name:
            ops.sigmoid_gate(o, full[:, self.gate_at:self.gate_at + H * V])
        return self.o(o, out_dtype=torch.float32 if self.out_float32 else None)

    @staticmethod
    def _single_rows(ctx: StepContext):
        """(first row, end) of the requests that bring one token, with what lies between them.  (In a captured graph they are the
        batch's last places.)"""
        if "single_rows" not in ctx.derived:
            cu = ctx.cu_seqlens_host
            rows = [cu[i] for i in range(len(cu) - 1) if cu[i + 1] - cu[i] == 1]
            ctx.derived["single_rows"] = (rows[0], rows[-1] + 1)
        return ctx.derived["single_rows"]

    # rows up to which the per-head products run on this package's own kernel (each weight read once, 32-bit
    # multiply-adds); beyond, bfloat16 goes to the library's batched product like the other prompt-sized products
    OWN_ABSORB_ROWS = 32

    def absorb(self, a, w, out) -> None:
        """out[:, h] = a[:, h] @ w[h]^T for every head (a [T, H, K], w [H, N, K], out [T, H, N], any strides)."""
        if a.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and a.shape[0] > self.OWN_ABSORB_ROWS:
            add_launches(1)
            torch.bmm(a.transpose(0, 1), w.transpose(1, 2), out=out.transpose(0, 1))
        else:
            ops.gemm_f32_batched(a, w, out)

    # What the two ways of a portion cost.  Absorbed: flops a second (mma.sync; 120 to 160e12 measured at R 512, 100e12 at
    # R 256, hence the 100 columns that _expanded_shape adds), bytes a second and seconds that its two products take whatever
    # the portion.  Expanded: flops a second of the product, bytes a second of the gather, seconds a CTA of the attention takes
    # for a tile of 128 keys with one and with both of its row tiles.
    RATES = (150e12, 6e11, 6e-6, 1000e12, 3e12, 1.8e-6, 2.85e-6)
    # Beside decoded tokens the expanded way's launches come on top of the absorbed one's.  Kernel by kernel that is so much more
    # of the host (s), which such a step is waiting for: 200 us a layer and 258 on the machine that was measured.
    MIXED_HOST = 76e-6
    # the keys and values of a step's portions, all heads, are expanded at once up to so many bytes
    EXPANDED_BYTES = 256 << 20
    _sms = 0                                                # of the device, asked at the first step that weighs the two

    def _expanded(self, ctx: StepContext, dtype):
        """Whether the step's portions run over expanded latents: None, or (rows of the gathered latents, row-tile pairs).  The
        absorbed form needs H (2 R + P) multiply-adds a (token, key) pair, the expanded one H (D + P + V) and R H (D + V) a key.
        But a CTA of the expanded attention walks all keys of its 256 rows one tile after the other, so a few rows behind a
        long history are the absorbed form's.  A layer of 16 heads of 128 + 64, R 512, absorbed and expanded (us): a prompt of
        64 tokens 51 and 37, of 2048 566 and 126; 64 tokens behind 4000 129 and 89, behind 8000 177 and 140, behind 16000 287 and
        232; 32 behind 16000 225 and 234; 256 behind 16000 1187 and 305; 8 heads of 64 + 32, R 256: 64 behind 4000 59 and 60, behind
        16000 115 and 155, 256 behind 16000 304 and 183.  (Two CTAs share a long walk where SMs are left over, which the rule does
        not know: it charges a walk to one, and keeps 64 tokens behind 8000 and more, and 256 of the small layer's, absorbed.)
        With decoded tokens in the step the absorbing products run for them all the same, and its launches too: nothing but the
        portions' attention is saved.  Eight tokens at 1000 beside a prompt, the same layer, as a graph and kernel by kernel:
        128 tokens 90 and 71, 172 and 247; 600 158 and 93, 175 and 247; 1024 263 and 109, 278 and 248; 2048 577 and 162, 589
        and 251; 64 behind 4000 161 and 135, 176 and 249; 256 behind 2000 211 and 112, 224 and 248; behind 4000 323 and 155, 337
        and 248.
        In a captured graph the lengths are bounds: the tokens spread evenly over the prompt places without a history for what
        the absorbed form costs at least, every place as long as it may get for what the other one costs at most."""
        if self.ukv is None or dtype != torch.bfloat16 or not ctx.any_prefill or not ctx.cu_seqlens_host:
            return None
        if ctx.any_decode and not latent_ops.tc_supported(dtype, self.R, self.P):
            return None                                      # the plain kernel for the single tokens does all rows at once
        key = ("latent_expanded", self.H, self.D, self.P, self.V, self.R, self.window)
        if key not in ctx.derived:
            ctx.derived[key] = self._expanded_shape(ctx)
        return ctx.derived[key]

    def _expanded_shape(self, ctx: StepContext):
        cu, window = ctx.cu_seqlens_host, int(self.window or 0)
        flops, weight_rate, products, expanding, gather, one, both = self.RATES
        H, D, P, V, R = self.H, self.D, self.P, self.V, self.R
        if ctx.decode_splits:                                # captured: any place may hold any of the prompt tokens
            lens = [b - a for a, b in zip(cu, cu[1:])]
            tokens, places = sum(n for n in lens if n != 1), sum(n != 1 for n in lens)
            if not tokens:
                return None
            longest = ctx.max_prefill_seq_len or ctx.max_seq_len
            bound = [(min(tokens, longest), longest)] * places
            pairs = tokens * tokens / (2.0 * places)
            tiles = tokens // 256 + places
            seen = [(tiles, 256, longest)]                   # (CTAs a head, rows of one, keys it walks) at most
        else:
            tokens, pairs, tiles, bound, seen, start = 0, 0, 0, [], [], 0
            for end, s in zip(cu[1:], ctx.seq_lens_host):    # (one turn over the requests: the host waits for it)
                n = end - start
                start = end
                if n <= 1:
                    continue
                count = (n + 255) // 256
                tokens += n
                pairs += n * (min(s - n, window) if window else s - n) + n * (n + 1) // 2
                tiles += count
                bound.append((n, s))
                seen.append((count, n, s - n // 2 if n > 256 else s))
            if not bound:
                return None
        if window:
            pairs = min(pairs, float(window) * tokens)
            seen = [(count, n, min(keys, window + 256)) for count, n, keys in seen]
        absorbed = pairs * H * 2 * (2 * R + P + 100) / flops
        if not ctx.any_decode:
            absorbed += H * R * (D + V) * 2 / weight_rate + products
        elif not ctx.decode_splits:
            absorbed -= self.MIXED_HOST
        longest_walk = walked = 0.0
        for count, n, keys in seen:
            walk = (keys + 127) // 128 * (both if n > 128 else one)
            longest_walk = max(longest_walk, walk)
            walked += count * walk
        if absorbed <= longest_walk:
            return None
        self._sms = self._sms or num_sms()
        rows = latent_ops.expanded_rows(bound, window)
        expanded = rows * R * H * 2 * (D + V) / expanding + rows * (R + P) * 4 / gather + max(longest_walk, H * walked / self._sms)
        if absorbed <= expanded or rows * H * (D + V) * 2 > self.EXPANDED_BYTES or tiles > 65535:
            return None
        return rows, tiles

    def attend_expanded(self, q, o, kv, g, ctx: StepContext, table, rows: int, tiles: int) -> None:
        window = int(self.window or 0)
        latent_ops.latent_q_turn(q, ctx.positions, table, self.H, self.D, self.P, halves=self.halves)
        latents = latent_ops.latent_rows(kv, g.block_table, ctx.cu_seqlens, ctx.seq_lens, rows, window)
        expanded = self.ukv(latents[:, :self.R])
        latent_ops.attention_latent_umma(q, o, latents, expanded, ctx.cu_seqlens, ctx.seq_lens, self.R, self.P, self.D,
                                         self.scale, window, sinks=self.sinks, pair_bound=tiles,
                                         max_keys=min(ctx.max_seq_len, rows))

    def attend(self, q_lat, o_lat, kv, g, ctx: StepContext, singles: bool = False) -> None:
        window = int(self.window or 0)
        if latent_ops.tc_supported(q_lat.dtype, self.R, self.P, g.block_size):
            # inside a captured graph the longest request is whatever the engine admits
            longest = self.env.max_positions if ctx.decode_splits else ctx.max_seq_len
            latent_ops.attention_latent_tc(q_lat, o_lat, kv, g.block_table, ctx.cu_seqlens, ctx.seq_lens, self.R, self.P,
                                           self.scale, window, max_q_len=ctx.max_q_len, max_seq_len=longest,
                                           sinks=self.sinks, singles=singles)
        else:
            latent_ops.attention_latent_generic(q_lat, o_lat, kv, g.block_table, ctx.cu_seqlens, ctx.positions, self.R,
                                                self.P, self.scale, window, sinks=self.sinks)
