"""The caller of the fused epilogue: a tensor-parallel Llama-style decoder for inference.

Mirrors the structure of the reference's ``model/transformer_model.py:397-811`` (``ModelArgs``,
``Attention`` with grouped-query heads, interleaved-pair RoPE and a KV cache, SwiGLU
``FeedForward``, pre-norm ``TransformerBlock``) and ``model/tensor_parallel.py:34-123``
(column-parallel ``wq/wk/wv/w1/w3``, row-parallel ``wo/w2``), with the one change the fused
operator exists for: a row-parallel projection returns its *partial* sums, and

    h, normed, scale = env.allreduce_add_rms_fused(partial, h, next_norm.weight, eps, fp8_out)

replaces ``reduce_from_tensor_parallel_region`` + ``x + ...`` + the following ``RMSNorm``
(``tensor_parallel.py:117-118``, ``transformer_model.py:610-618``) at both sites of every
layer.  With ``fp8=True`` the normalised activations leave the operator as FP8-e4m3 with one
scale per token, and the column-parallel projections that consume them run as FP8 GEMMs with
row-wise scales: for decode batches of up to 32 tokens this library's own weight-streaming kernels
(``gpuk_b200.fp8_linear``, ``csrc/fp8_linear.cu`` and ``csrc/stream_linear.cu``; the row-parallel projections in bf16 likewise),
otherwise ``torch._scaled_mm`` (a library GEMM; ``own_fp8_gemm=False`` uses libraries everywhere).  Both give the same results to
within one bf16 step.

``fused=False`` runs the reference arrangement on the same weights -- NCCL ``all_reduce``, then
add, RMSNorm (and quantisation) as separate PyTorch operators -- and is the comparison arm.

Fix-ups relative to the reference, which cannot run with more than one rank as it stands
(``WorkerProc.__call__`` raises, ``:788-789``): the KV cache holds this rank's KV heads only
(the reference sizes it with the global count, ``:674``), weights are random-initialised per
shard on the device, and nothing is compiled or traced.
"""
from __future__ import annotations

import math
from dataclasses import dataclass
from typing import List, Optional, Tuple

import torch
import torch.distributed as dist
import torch.nn.functional as F

import gpuk_b200 as gpuk
from gpuk_b200 import _native


@dataclass
class DecoderArgs:
    """Subset of the reference's ``ModelArgs`` (``transformer_model.py:419-443``) a dense decoder needs."""
    dim: int = 8192
    n_layers: int = 4
    n_heads: int = 64
    n_kv_heads: int = 8
    head_dim: int = 128
    ffn_dim: int = 28672
    vocab_size: int = 32768
    max_seq_len: int = 2304
    norm_eps: float = 1e-6
    rope_theta: float = 500000.0
    dtype: torch.dtype = torch.bfloat16


def _shard_rows(master: torch.Tensor, rank: int, world: int) -> torch.Tensor:
    """Column-parallel shard: rows [rank*n/world, (rank+1)*n/world) of a [out, in] weight (``tensor_parallel.py:24-30``)."""
    n = master.shape[0] // world
    return master[rank * n:(rank + 1) * n].contiguous()


def _shard_cols(master: torch.Tensor, rank: int, world: int) -> torch.Tensor:
    """Row-parallel shard: columns of a [out, in] weight."""
    n = master.shape[1] // world
    return master[:, rank * n:(rank + 1) * n].contiguous()


def _xavier(out_f: int, in_f: int, gen: torch.Generator, device, dtype) -> torch.Tensor:
    std = math.sqrt(2.0 / (in_f + out_f))     # init.xavier_normal_ on the full matrix (tensor_parallel.py:62-67)
    return (torch.randn(out_f, in_f, generator=gen, device=device, dtype=torch.float32) * std).to(dtype)


class _Linear:
    """y = x @ W^T for one shard, in the activation dtype or as an FP8 GEMM with row-wise scales."""

    def __init__(self, weight: torch.Tensor, fp8: bool, own_gemm: bool = True):
        self.weight = weight                                  # [out_local, in]
        self.fp8 = fp8
        self.own_gemm = own_gemm                              # decode batches: this library's weight-streaming kernels
        self.w_packed = None                                  # ... and a blocked copy of FP8 weights, made at first use
        if fp8:
            amax = weight.float().abs().amax(dim=1, keepdim=True).clamp_(min=1e-12)
            self.w_scale = (amax / 448.0).t().contiguous()    # [1, out_local] fp32, one scale per output channel
            self.w_q = (weight.float() / amax * 448.0).clamp_(-448, 448).to(torch.float8_e4m3fn)   # [out, in] row-major

    def streamed(self, x: torch.Tensor):
        """The weight and its scales (None in bf16) as the streaming kernels with a fused epilogue take them, or None where the projection runs
        elsewhere: on the CPU, in a library, or -- 8 tokens at most on small FP8 weights, up to where the epilogue repays the time by which the
        streaming kernel is behind -- on the warp-level kernel (csrc/fp8_linear.cu)."""
        w = self.w_q if self.fp8 else self.weight
        if not (self.own_gemm and x.is_cuda and 0 < x.shape[0] <= 32 and self.weight.dtype == torch.bfloat16 and x.dtype == w.dtype):
            return None
        if w.shape[0] % 128 or w.shape[1] % (64 if self.fp8 else 8) or (self.fp8 and x.shape[0] <= 8 and w.numel() <= 12 << 20):
            return None
        return w, (self.w_scale if self.fp8 else None)

    def __call__(self, x: torch.Tensor, x_scale: Optional[torch.Tensor] = None) -> torch.Tensor:
        # up to 32 tokens: the streaming kernels, faster than the library on FP8 weights and on large or narrow bf16 ones, within a microsecond and a half of it
        # elsewhere (stream_linear.cu), with 4 us less on the host for a call
        own = self.own_gemm and x.is_cuda and 0 < x.shape[0] <= 32 and self.weight.dtype == torch.bfloat16
        if self.fp8 and x.dtype == torch.float8_e4m3fn:
            if own and _native.no_modes() and (x.shape[0] <= 8 or self.w_q.is_contiguous()):
                if gpuk.fp8_linear_supported(x.shape[0], *self.w_q.shape):
                    if x.shape[0] > 8:
                        return gpuk.fp8_linear(x, x_scale, self.w_q, self.w_scale)
                    # up to 8 tokens blocked weights are 3 to 12 % faster (2048 x 5120: 4.9 / 5.7 us), beyond within 2 % of row-major ones
                    if self.w_packed is None:
                        self.w_packed = gpuk.fp8_pack_weight(self.w_q)
                    return gpuk.fp8_linear(x, x_scale, self.w_packed, self.w_scale, packed=True)
            return torch._scaled_mm(x, self.w_q.t(), scale_a=x_scale, scale_b=self.w_scale, out_dtype=self.weight.dtype)
        if own and x.dtype == torch.bfloat16 and self.weight.shape[0] % 128 == 0 and self.weight.shape[1] % 8 == 0:
            y = _native.linear(x, self.weight)
            if y is not None:      # weights that are views, and modes that want to see operators, belong to the library
                return y
        return F.linear(x, self.weight)


class TPDecoder:
    """Random-initialised decoder, sharded over the ranks of ``env``'s group; inference only."""

    def __init__(self, args: DecoderArgs, env, *, device, fused: bool = True, fp8: bool = True, seed: int = 1234,
                 master_init: bool = False, max_batch: int = 32, own_fp8_gemm: bool = True):
        self.args, self.env, self.device, self.fused, self.fp8 = args, env, torch.device(device), fused, fp8
        self.rank, self.world = env.rank, env.world_size
        a, w, r = args, self.world, self.rank
        assert a.n_heads % w == 0 and a.n_kv_heads % w == 0 and a.ffn_dim % w == 0, "heads and FFN must divide over the ranks"
        self.h_local, self.kv_local = a.n_heads // w, a.n_kv_heads // w
        hd = a.head_dim

        def make(out_f, in_f, tag, split):
            """One weight shard.  master_init draws the full matrix (identical on all ranks, as the
            reference does on the CPU) and slices it; otherwise the shard is drawn directly."""
            if master_init:
                g = torch.Generator(device="cpu").manual_seed(seed * 1000 + tag)
                m = _xavier(out_f, in_f, g, "cpu", a.dtype)
                s = _shard_rows(m, r, w) if split == "rows" else (_shard_cols(m, r, w) if split == "cols" else m)
                return s.to(self.device)
            g = torch.Generator(device=self.device).manual_seed(seed * 1000 + tag * 16 + (r if split else 0))
            so, si = (out_f // w, in_f) if split == "rows" else ((out_f, in_f // w) if split == "cols" else (out_f, in_f))
            std_w = _xavier(so, si, g, self.device, torch.float32) * (math.sqrt(so + si) / math.sqrt(out_f + in_f))
            return std_w.to(a.dtype)

        self.tok_embeddings = make(a.vocab_size, a.dim, 1, None)
        self.layers: List[dict] = []
        for li in range(a.n_layers):
            t = 100 * (li + 1)
            wq = make(a.n_heads * hd, a.dim, t + 1, "rows")
            wk = make(a.n_kv_heads * hd, a.dim, t + 2, "rows")
            wv = make(a.n_kv_heads * hd, a.dim, t + 3, "rows")
            w1 = make(a.ffn_dim, a.dim, t + 5, "rows")
            w3 = make(a.ffn_dim, a.dim, t + 6, "rows")
            norm_gen = torch.Generator(device="cpu").manual_seed(seed * 1000 + t + 8)
            self.layers.append({
                # one GEMM for q|k|v and one for w1|w3: they share their input
                "wqkv": _Linear(torch.cat([wq, wk, wv], 0), fp8, own_fp8_gemm),
                "wo": _Linear(make(a.dim, a.n_heads * hd, t + 4, "cols"), False, own_fp8_gemm),
                "w13": _Linear(torch.cat([w1, w3], 0), fp8, own_fp8_gemm),
                "w2": _Linear(make(a.dim, a.ffn_dim, t + 7, "cols"), False, own_fp8_gemm),
                "attention_norm": (1 + 0.1 * torch.randn(a.dim, generator=norm_gen)).to(a.dtype).to(self.device),
                "ffn_norm": (1 + 0.1 * torch.randn(a.dim, generator=norm_gen)).to(a.dtype).to(self.device),
                "k_cache": torch.zeros(max_batch, self.kv_local, a.max_seq_len, hd, dtype=a.dtype, device=self.device),
                "v_cache": torch.zeros(max_batch, self.kv_local, a.max_seq_len, hd, dtype=a.dtype, device=self.device),
            })
        norm_gen = torch.Generator(device="cpu").manual_seed(seed * 1000 + 9)
        self.norm = (1 + 0.1 * torch.randn(a.dim, generator=norm_gen)).to(a.dtype).to(self.device)
        self.output = _Linear(make(a.vocab_size, a.dim, 2, "rows"), fp8, own_fp8_gemm)
        inv = 1.0 / (a.rope_theta ** (torch.arange(0, hd, 2, dtype=torch.int64).float() / hd))   # :497-502
        freqs = torch.outer(torch.arange(a.max_seq_len * 2, dtype=torch.float32), inv)
        self.cos, self.sin = freqs.cos().to(self.device), freqs.sin().to(self.device)
        self._zeros = {}
        # the elementwise steps between the projections as this library's kernels (csrc/decoder_ops.cu)
        self.own_elementwise = fused and self.device.type == "cuda" and a.dtype == torch.bfloat16 and hd % 16 == 0 and a.ffn_dim // w % 8 == 0
        # ... and so attention over the cache, for one new token per sequence (csrc/attention.cu) and for more (csrc/prefill_attention.cu)
        self.own_attention = hd == 128 and self.h_local % self.kv_local == 0

    # ------------------------------------------------------------------------------------
    def fill_kv_cache(self, upto: int, seed: int = 7) -> None:
        """Seeded N(0,1) keys and values for positions [0, upto): stands in for a prefill."""
        for li, layer in enumerate(self.layers):
            g = torch.Generator(device=self.device).manual_seed(seed * 100 + li * 16 + self.rank)
            for name in ("k_cache", "v_cache"):
                c = layer[name]
                c[:, :, :upto] = torch.randn(c.shape[0], c.shape[1], upto, c.shape[3], generator=g, device=self.device,
                                             dtype=torch.float32).to(c.dtype)

    def _rope(self, x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> torch.Tensor:
        """Interleaved pairs in, halves out (``transformer_model.py:504-519``, rope_interval_split)."""
        x1, x2 = x[..., 0::2], x[..., 1::2]
        cos, sin = cos.unsqueeze(-2), sin.unsqueeze(-2)
        return torch.cat((x1 * cos - x2 * sin, x2 * cos + x1 * sin), dim=-1).type_as(x)

    def _norm_only(self, h: torch.Tensor, weight: torch.Tensor):
        """RMSNorm (+ FP8) of the embeddings before the first layer: the fused operator with a
        zero residual on this rank alone."""
        if self.fused:
            z = self._zeros.get(h.shape)
            if z is None:
                z = self._zeros[h.shape] = torch.zeros_like(h)
            results = _native.add_rms(0, h, z, weight, self.args.norm_eps, 3 if self.fp8 else 0, None)
            if results is not None:
                return results[1], results[2] if self.fp8 else None
            residual_out = torch.empty_like(h)
            if self.fp8:
                normed = torch.empty(h.shape, dtype=torch.float8_e4m3fn, device=h.device)
                scale = torch.empty(h.shape[0], 1, dtype=torch.float32, device=h.device)
                gpuk.allreduce_rms(0, h, z, weight, residual_out, normed, scale, self.args.norm_eps, 3)
                return normed, scale
            normed = torch.empty_like(h)
            scale = torch.empty(1, dtype=torch.float32, device=h.device)
            gpuk.allreduce_rms(0, h, z, weight, residual_out, normed, scale, self.args.norm_eps, 0)
            return normed, None
        return self._unfused_norm(h, weight)

    def _unfused_norm(self, h, weight):
        v = h.float().pow(2).mean(-1, keepdim=True)
        n = weight * (h * torch.rsqrt(v + self.args.norm_eps)).to(h.dtype)
        if not self.fp8:
            return n, None
        scale = n.float().abs().amax(dim=-1, keepdim=True) / 448.0
        return (n.float() / scale).clamp_(-448, 448).to(torch.float8_e4m3fn), scale

    def _reduce_add_norm(self, partial, h, weight) -> Tuple[torch.Tensor, torch.Tensor, Optional[torch.Tensor]]:
        """all-reduce(partial) + h -> new h; RMSNorm(new h) * weight (-> FP8) -> input of the next projections."""
        if self.fused:
            h, normed, scale = self.env.allreduce_add_rms_fused(partial, h, weight, self.args.norm_eps, self.fp8)
            return h, normed, (scale if self.fp8 else None)
        if self.world > 1:
            dist.all_reduce(partial, group=self.env.group)       # tensor_parallel.py:118
        h = h + partial                                          # transformer_model.py:611,617
        normed, scale = self._unfused_norm(h, weight)            # :466-471
        return h, normed, scale

    @torch.no_grad()
    def forward(self, tokens: torch.Tensor, input_pos: torch.Tensor, cache_len: Optional[int] = None) -> torch.Tensor:
        """tokens [b, t] at positions input_pos [t] (KV cache updated in place) -> logits [b, t, vocab/world]
        of this rank's vocabulary shard.  cache_len = last position + 1; pass it to avoid a device read.

        A position outside the cache is refused where it can be seen without a device read of its own (positions on the host, or no
        cache_len).  Elsewhere this library's kernels write neither its key nor its value, its token's logits are NaN, and
        ``gpuk_fp8_linear_status`` reports it."""
        a = self.args
        b, t = tokens.shape
        hd = a.head_dim
        h = F.embedding(tokens, self.tok_embeddings).view(b * t, a.dim)
        # positions in any other form that indexes a tensor go to the operators, as do caches, tables and weights that the kernels cannot read as they are
        own = self.own_elementwise and isinstance(input_pos, torch.Tensor) and input_pos.shape == (t,)
        if own:
            pos = input_pos.to(device=self.device, dtype=torch.int64).contiguous()
            own = pos is input_pos or (input_pos.dtype in (torch.int64, torch.int32) and (not input_pos.is_cuda or input_pos.device == self.cos.device))
        here = input_pos
        if own and input_pos.is_cuda:
            here = input_pos.cpu() if cache_len is None else None
        last = int(here[-1]) + 1 if cache_len is None else cache_len
        if own:
            if last > a.max_seq_len and t == 1 and cache_len is not None:
                last = a.max_seq_len      # as a slice of the cache takes it
            if last > a.max_seq_len:
                raise RuntimeError(f"position {last - 1} is beyond the KV cache ({a.max_seq_len} positions)")
            if here is not None and t:
                lo, hi = map(int, here.aminmax())
                if lo < -a.max_seq_len or hi >= a.max_seq_len:
                    raise RuntimeError(f"a position in [{lo}, {hi}] is beyond the KV cache ({a.max_seq_len} positions)")
        tables = mask = None      # what the operators need, once one of them is called
        normed, scale = self._norm_only(h, self.layers[0]["attention_norm"])
        for li, layer in enumerate(self.layers):
            q = att = act = None      # a native call returns None where the operators are wanted
            fused = layer["wqkv"].streamed(normed) if own and hd == 128 else None
            if fused is not None:
                q = _native.qkv_rope(normed, scale, *fused, self.cos, self.sin, pos, layer["k_cache"], layer["v_cache"], self.h_local)
            if q is None:
                qkv = layer["wqkv"](normed, scale)
                if own:
                    q = _native.rope_append(qkv, self.cos, self.sin, pos, layer["k_cache"], layer["v_cache"], self.h_local)
            if q is not None:
                q = q.view(b, t, self.h_local, hd)
            else:
                if tables is None:
                    tables = self.cos[input_pos], self.sin[input_pos]
                q, k, v = qkv.view(b, t, self.h_local + 2 * self.kv_local, hd).split([self.h_local, self.kv_local, self.kv_local], dim=2)
                q, k = self._rope(q, *tables), self._rope(k, *tables)
                layer["k_cache"][:b, :, input_pos] = k.transpose(1, 2)
                layer["v_cache"][:b, :, input_pos] = v.transpose(1, 2)
            if own and self.own_attention and last >= 1:
                if t > 1:
                    att = _native.prefill_attention(q, layer["k_cache"], layer["v_cache"], pos, last)
                elif self.h_local // self.kv_local <= 16 and (last <= 32768 or b * self.kv_local > 16):
                    # Up to 16 pairs of sequence and kv head, the eight parts that a pair's keys are cut into leave SMs idle, and the library's attention, which cuts further, is
                    # ahead on the device for long contexts (one pair: 4096 keys 8.1 / 7.3 us, 16384 20.3 / 9.5, 32768 35.9 / 11.5; eight: 32768 37.8 / 25.5).  Its call costs
                    # 25 us more on the host, so it is taken where that is made good.
                    att = _native.decode_attention(q.view(b, self.h_local, hd), layer["k_cache"], layer["v_cache"], last)
            if att is None:
                if t > 1 and mask is None:
                    mask = (torch.arange(last, device=self.device)[None, :] <= input_pos[:, None])[None, None]
                    if own:
                        mask = mask | (input_pos < -a.max_seq_len)[:, None]      # a token that the rotary embedding marked attends, and stays marked
                att = F.scaled_dot_product_attention(q.transpose(1, 2), layer["k_cache"][:b, :, :last], layer["v_cache"][:b, :, :last],
                                                     attn_mask=mask, enable_gqa=True).transpose(1, 2).reshape(b * t, self.h_local * hd)
            partial = layer["wo"](att)
            h, normed, scale = self._reduce_add_norm(partial, h, layer["ffn_norm"])
            fused = layer["w13"].streamed(normed) if own else None
            if fused is not None:
                act = _native.swiglu(normed, scale, *fused)
            if act is None:
                f13 = layer["w13"](normed, scale)
                if own:
                    act = _native.silu_mul(f13)
            if act is None:
                f1, f3 = f13.split(a.ffn_dim // self.world, dim=-1)
                act = F.silu(f1) * f3
            partial = layer["w2"](act)
            nxt = self.layers[li + 1]["attention_norm"] if li + 1 < a.n_layers else self.norm
            h, normed, scale = self._reduce_add_norm(partial, h, nxt)
        return self.output(normed, scale).view(b, t, -1)
