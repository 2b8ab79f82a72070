"""One decode step of a pre-norm decoder stack with fp8-e4m3 linears -- the shape of xn-moshi's
BatchedTransformerLayer (xn-moshi/src/batched_transformer.rs:92-199, 246-268) with the gated FFN of
xn-moshi/src/transformer.rs:234-247, restricted to what the benchmark's decoder configuration lists:
RMSNorm -> fused qkv projection -> KV append -> attention over a (streams, heads, context, 128) bf16
cache -> output projection -> residual -> RMSNorm -> gated SiLU FFN -> residual.  No rope (the
configuration does not list it).  T = 1 token per stream per step; streams are independent, which is
what lets them be sharded over GPUs with no communication.

Every operation is a call into libxn_mm.so on the current torch stream, so a step can be captured in
a CUDA graph.  Buffers are allocated once in the constructor.
"""
from __future__ import annotations

import torch

from . import _host
from ._lib import lib


class DecoderStack:
    def __init__(self, n_layers: int, d_model: int, n_heads: int, ffn_hidden: int, streams: int, context: int,
                 device, eps: float = 1e-5, seed: int = 4, variant: int = 0, kv_init: str = "normal",
                 attention: str = "separate"):
        """attention: how a layer's cache append, attention, merge of the context slices and e4m3 split are launched.
        "separate" = xn_mm_kv_append2 + xn_mm_decode_attention_split_e4m3 (three launches; the fastest at 32 streams x
        3000 tokens), "fused" = xn_mm_decode_attention_append_e4m3 (one or two launches, the library decides where the
        merge runs), "fused_one_launch" = the same with the merge forced into the attention kernel.  All three give
        identical results."""
        assert d_model == n_heads * 128, "head_dim is 128"
        assert attention in ("separate", "fused", "fused_one_launch")
        self.attention = attention
        self.L, self.d, self.H, self.hid, self.B, self.ctx = n_layers, d_model, n_heads, ffn_hidden, streams, context
        self.eps, self.variant, self.dev = eps, variant, device
        g = torch.Generator(device=device).manual_seed(seed)
        from .ops import quantize_weights_fp8

        def qlin(n, k):
            w = torch.randn(n, k, generator=g, device=device) * 0.02
            q = quantize_weights_fp8(w)
            del w
            return q

        self.layers = []
        for _ in range(n_layers):
            lay = {
                "norm1": torch.ones(d_model, device=device, dtype=torch.bfloat16),
                "norm2": torch.ones(d_model, device=device, dtype=torch.bfloat16),
                "in_proj": qlin(3 * d_model, d_model),
                "out_proj": qlin(d_model, d_model),
                "linear_in": qlin(2 * ffn_hidden, d_model),
                "linear_out": qlin(d_model, ffn_hidden),
            }
            shape = (streams, n_heads, context, 128)
            if kv_init == "normal":
                lay["k"] = torch.randn(shape, generator=g, device=device, dtype=torch.bfloat16)
                lay["v"] = torch.randn(shape, generator=g, device=device, dtype=torch.bfloat16)
            else:
                lay["k"] = torch.zeros(shape, device=device, dtype=torch.bfloat16)
                lay["v"] = torch.zeros(shape, device=device, dtype=torch.bfloat16)
            self.layers.append(lay)
        B, d, hid = streams, d_model, ffn_hidden
        kmax = max(d, hid)
        u8 = dict(dtype=torch.uint8, device=device)
        bf = dict(dtype=torch.bfloat16, device=device)
        self.hi, self.lo = torch.empty(B * kmax, **u8), torch.empty(B * kmax, **u8)
        self.xs = torch.empty(B, dtype=torch.float32, device=device)
        self.qkv = torch.empty(B, 3 * d, **bf)
        self.attn = torch.empty(B, d, **bf)
        # (maximum, sum, output) records of the context slices of the attention
        self.attn_ws_bytes = int(lib().xn_mm_decode_attention_append_workspace_bytes(B, n_heads, context))
        self.attn_ws = torch.empty(self.attn_ws_bytes, dtype=torch.uint8, device=device)
        self.proj = torch.empty(B, d, **bf)
        self.h = torch.empty(B, 2 * hid, **bf)
        self.x_mid = torch.empty(B, d, **bf)
        self.x_out = torch.empty(B, d, **bf)
        self.pos = torch.full((B,), context - 1, dtype=torch.int64, device=device)
        self.mask = None  # optional f32 [B, context] additive mask

    def step(self, x: torch.Tensor) -> torch.Tensor:
        """x: [streams, d_model] bf16 (the embedded token of every stream). Returns the stack's output.

        Per layer: [norm1 + split] -> in_proj -> cache append, attention, merge + split -> out_proj -> add + norm2 + split
        -> linear_in -> silu * mul + split -> linear_out -> add + next norm1 + split; the walk over the layers is native
        (csrc/host/binding.cpp, decoder_step)."""
        return _host.decoder_step(self, x)

    def bytes_per_step(self) -> dict:
        d, hid, B, ctx, H = self.d, self.hid, self.B, self.ctx, self.H
        w = self.L * (3 * d * d + d * d + 2 * hid * d + d * hid + 4 * (3 * d + d + 2 * hid + d))
        kv = self.L * 2 * B * H * ctx * 128 * 2
        return {"weights": w, "kv": kv, "total": w + kv}

    def launches_per_step(self) -> int:
        # per layer: in_proj, cache append + attention + merge of the context slices with the e4m3 split (three launches,
        # two or one, see `attention`), out_proj, add+norm, linear_in, silu*mul, linear_out, add+norm (plain add after the last layer); one norm
        # up front
        per_layer = 10 if self.attention == "separate" else (8 if self._merge_in_kernel() else 9)
        return self.L * per_layer + 1

    def _merge_in_kernel(self) -> bool:
        """The library's policy (xn_mm_decode_attention_append_e4m3): the merge of the context slices runs inside the
        attention kernel when a resident slot sees at most two CTAs, otherwise as its own launch."""
        if self.attention == "fused_one_launch":
            return True
        ctas = self.attn_ws_bytes // (130 * 4)  # one 130-float record per (stream, head, slice)
        sms = torch.cuda.get_device_properties(self.dev).multi_processor_count
        return ctas <= sms * 5 * 2
