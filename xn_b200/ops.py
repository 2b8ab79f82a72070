"""Host-side mirror of xn's matmul interface over the C ABI.

Names and argument meaning follow the reference: ``matmul`` / ``matmul_t`` / ``matmul_with_t``
(xn-core/src/ops.rs:631-714), the in-place ``matmul_`` (xn-core/src/inplace_ops.rs:318-436) and
``Linear`` (xn-core/src/nn/linear.rs:4-71).  A ``torch.Tensor`` on a CUDA device plays the role of
xn's ``Tensor`` / ``TensorView``: its storage pointer, ``storage_offset()``, ``stride()`` and
``shape`` are exactly the (storage, start_offset, strides, dims) a TensorView carries
(xn-core/src/tensor_view.rs:103-109), so transposed / narrowed views reach the kernels zero-copy.
torch is used for device memory and streams only; all arithmetic happens in libxn_mm.so.  The operators a model calls
per token go through the native host module (csrc/host/binding.cpp); the rest binds the library with ctypes.
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _host, _lib
from ._lib import BF16, F16, F32, XnError, check, lib

_DT = {torch.float32: F32, torch.float16: F16, torch.bfloat16: BF16}


def _dtype_code(t: torch.Tensor) -> int:
    if t.dtype not in _DT:
        # the reference refuses other element types at the same point (cuda_backend.rs:862)
        raise XnError(_lib.ERR_UNSUPPORTED, f"GEMM not supported for dtype {t.dtype}")
    return _DT[t.dtype]


def _stream() -> C.c_void_p:
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _require_cuda(*ts: torch.Tensor) -> None:
    for t in ts:
        if not t.is_cuda:
            raise XnError(_lib.ERR_INVALID, "xn_b200 runs on CUDA tensors only; there is no CPU path")


def _base_ptr(t: torch.Tensor) -> int:
    return t.untyped_storage().data_ptr()


def _arr(vals):
    return (C.c_size_t * len(vals))(*[int(v) for v in vals])


def matmul_plan(lhs: torch.Tensor, rhs: torch.Tensor, rhs_t: bool, dst_capacity: int):
    """The 12 ``Backend::gemm`` arguments for two views (xn_mm_matmul_plan)."""
    out = (C.c_size_t * 12)()
    check(lib().xn_mm_matmul_plan(lhs.dim(), _arr(lhs.shape), _arr(lhs.stride()), rhs.dim(), _arr(rhs.shape),
                                  _arr(rhs.stride()), int(rhs_t), dst_capacity, out))
    return [int(v) for v in out]


def gemm(dst: torch.Tensor, lhs: torch.Tensor, lhs_off: int, rhs: torch.Tensor, rhs_off: int, m, n, k, lhs_b,
         lhs_b_stride, rhs_b_stride, dst_strides, lhs_strides, rhs_strides) -> None:
    """``Backend::gemm`` on flat storages (xn-core/src/backend.rs:135-148)."""
    _require_cuda(dst, lhs, rhs)
    dt = _dtype_code(dst)
    check(lib().xn_mm_gemm(dt, dst.data_ptr(), lhs.data_ptr(), lhs_off, rhs.data_ptr(), rhs_off, m, n, k, lhs_b,
                           lhs_b_stride, rhs_b_stride, dst_strides[0], dst_strides[1], lhs_strides[0],
                           lhs_strides[1], rhs_strides[0], rhs_strides[1], _stream()))


def matmul_(dst: torch.Tensor, lhs: torch.Tensor, rhs: torch.Tensor, rhs_t: bool) -> None:
    """``Tensor::matmul_``: dst (a whole contiguous tensor) = lhs @ rhs or lhs @ rhs^T."""
    _host.matmul_(dst, lhs, rhs, rhs_t)


def matmul_causal_(dst: torch.Tensor, lhs: torch.Tensor, rhs: torch.Tensor, rhs_t: bool, mode: int, offset: int) -> None:
    """``matmul_`` for the two products of causal attention (xn_mm_gemm_causal): mode 1 = scores ``q @ k^T`` (tiles
    beyond the causal horizon are skipped and left unwritten), mode 2 = values ``p @ v`` (the masked tail of every
    row of p is not read).  Key j is visible to query row i iff j <= i + offset."""
    _require_cuda(dst, lhs, rhs)
    if not (dst.dtype == lhs.dtype == rhs.dtype):
        raise XnError(_lib.ERR_INVALID, f"matmul dtype mismatch: {dst.dtype}, {lhs.dtype}, {rhs.dtype}")
    dt = _dtype_code(dst)
    a = matmul_plan(lhs, rhs, rhs_t, dst.numel())
    check(lib().xn_mm_gemm_causal(mode, offset, dt, dst.data_ptr(), _base_ptr(lhs), lhs.storage_offset(), _base_ptr(rhs),
                                  rhs.storage_offset(), *a, _stream()))


def attention_prefill_(out: torch.Tensor, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float) -> None:
    """Causal attention over a block of query rows in one kernel (xn_mm_attention_prefill).  q: [heads, T, 128] view,
    k, v: [heads, context, 128] views with a common row pitch and head stride (e.g. the slices of a fused qkv projection
    viewed per head); out: [T, heads * 128] rows (row pitch out.stride(0)).  Key j is visible to row i iff
    j <= i + (context - T)."""
    _require_cuda(out, q, k, v)
    heads, t_rows, hd = q.shape
    ctx = k.shape[1]
    if not (q.dtype == k.dtype == v.dtype == out.dtype):
        raise XnError(_lib.ERR_INVALID, "attention_prefill: dtype mismatch")
    if not (q.stride(2) == k.stride(2) == v.stride(2) == 1 and q.stride(1) == k.stride(1) == v.stride(1)
            and q.stride(0) == k.stride(0) == v.stride(0) and out.stride(1) == 1):
        raise XnError(_lib.ERR_INVALID, "attention_prefill: q, k, v must share one row pitch and one head stride")
    es = q.element_size()
    check(lib().xn_mm_attention_prefill(_dtype_code(q), out.data_ptr(), out.stride(0),
                                        _base_ptr(q) + q.storage_offset() * es, _base_ptr(k) + k.storage_offset() * es,
                                        _base_ptr(v) + v.storage_offset() * es, q.stride(1), q.stride(0), heads, hd, t_rows, ctx,
                                        float(scale), _stream()))


def matmul_with_t(lhs: torch.Tensor, rhs: torch.Tensor, rhs_t: bool) -> torch.Tensor:
    """``ops::matmul_with_t``: output shape = lhs batch dims + [M, N], allocated uninitialised."""
    return _host.matmul_with_t(lhs, rhs, rhs_t)


def matmul(lhs: torch.Tensor, rhs: torch.Tensor) -> torch.Tensor:
    return _host.matmul_with_t(lhs, rhs, False)


def matmul_t(lhs: torch.Tensor, rhs: torch.Tensor) -> torch.Tensor:
    return _host.matmul_with_t(lhs, rhs, True)


class Linear:
    """``nn::Linear``: weight (out_features, in_features), optional bias (out_features)."""

    def __init__(self, weight: torch.Tensor, bias: torch.Tensor | None = None):
        self.weight, self.bias = weight, bias

    def with_bias(self, bias: torch.Tensor) -> "Linear":
        self.bias = bias
        return self

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        w, b = self.weight, self.bias
        y = _host.linear(x, w, b)
        if y is not None:
            return y
        y = matmul_t(x, w)  # views the Linear entry point does not take
        if b is not None:
            # the reference's separate broadcast_add (nn/linear.rs:61-64)
            check(lib().xn_mm_add_bias(_dtype_code(y), y.data_ptr(), y.data_ptr(), b.contiguous().data_ptr(),
                                       y.numel() // y.shape[-1], y.shape[-1], _stream()))
        return y

    __call__ = forward


# ---------------------------------------------------------------------------------------------
# Quantized linears (no counterpart in the reference): same forward(x) signature as Linear.
# ---------------------------------------------------------------------------------------------
def quantize_rows_i8(x: torch.Tensor, out: tuple[torch.Tensor, torch.Tensor] | None = None):
    """Per-row symmetric int8 quantization; `out` = (xq int8 [m,k], x_scale f32 [m]) reuses buffers."""
    xq, xs = out if out is not None else (None, None)
    return _host.quantize_rows_i8(x, xq, xs)


def quantize_weights_q4(w: torch.Tensor) -> torch.Tensor:
    """W [n,k] -> q4 tiles (uint8 buffer holding nibbles and block scales)."""
    _require_cuda(w)
    w = w.contiguous()
    n, k = w.shape
    packed = torch.empty(lib().xn_mm_q4_packed_bytes(n, k), dtype=torch.uint8, device=w.device)
    check(lib().xn_mm_quantize_weights_q4(packed.data_ptr(), w.data_ptr(), _dtype_code(w), n, k, _stream()))
    return packed


def linear_q4(xq: torch.Tensor, x_scale: torch.Tensor, wq_packed: torch.Tensor, n: int,
              partials: torch.Tensor | None = None, out: torch.Tensor | None = None) -> torch.Tensor:
    return _host.linear_block(4, xq, x_scale, wq_packed, n, partials, out)


def quantize_weights_q8(w: torch.Tensor) -> torch.Tensor:
    """W [n,k] -> q8 tiles (int8 block-quantized, scale = max|w|/127 per 32-block)."""
    _require_cuda(w)
    w = w.contiguous()
    n, k = w.shape
    packed = torch.empty(lib().xn_mm_q8_packed_bytes(n, k), dtype=torch.uint8, device=w.device)
    check(lib().xn_mm_quantize_weights_q8(packed.data_ptr(), w.data_ptr(), _dtype_code(w), n, k, _stream()))
    return packed


def linear_q8(xq: torch.Tensor, x_scale: torch.Tensor, wq_packed: torch.Tensor, n: int,
              partials: torch.Tensor | None = None, out: torch.Tensor | None = None) -> torch.Tensor:
    return _host.linear_block(8, xq, x_scale, wq_packed, n, partials, out)


class LinearQ4:
    """int4 block-quantized linear: forward(x) quantizes x per row to int8, returns f32."""

    def __init__(self, wq_packed, out_features: int, in_features: int):
        self.wq, self.n, self.k = wq_packed, out_features, in_features

    @classmethod
    def from_weight(cls, w: torch.Tensor) -> "LinearQ4":
        return cls(quantize_weights_q4(w), w.shape[0], w.shape[1])

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return _host.linear_q4_forward(x, self.wq, self.n, self.k)

    __call__ = forward

    def forward_host(self, x_host: torch.Tensor, y_host: torch.Tensor) -> torch.Tensor:
        """x_host [m,k] f32 and y_host [m,n] f32 in (pinned) host memory: one library call enqueues the copy in,
        the row quantizer, the linear and the copy out on the current stream (xn_mm_linear_q4_host); the result
        is valid after the stream has been synchronised.  Staging buffers are kept per batch size."""
        m = x_host.shape[0]
        if x_host.is_cuda or y_host.is_cuda or x_host.dtype != torch.float32 or y_host.dtype != torch.float32:
            raise XnError(_lib.ERR_INVALID, "forward_host takes float32 host tensors")
        if list(x_host.shape) != [m, self.k] or list(y_host.shape) != [m, self.n] or not x_host.is_contiguous() \
                or not y_host.is_contiguous():
            raise XnError(_lib.ERR_INVALID, f"forward_host: expected contiguous [{m},{self.k}] and [{m},{self.n}]")
        ws = self._host_ws.get(m) if hasattr(self, "_host_ws") else None
        if ws is None:
            if not hasattr(self, "_host_ws"):
                self._host_ws = {}
            ws = torch.empty(lib().xn_mm_linear_q4_host_workspace_bytes(m, self.n, self.k), dtype=torch.uint8,
                             device=self.wq.device)
            self._host_ws[m] = ws
        check(lib().xn_mm_linear_q4_host(y_host.data_ptr(), x_host.data_ptr(), self.wq.data_ptr(), m, self.n, self.k,
                                         ws.data_ptr(), ws.numel(), _stream()))
        return y_host


def quantize_weights_fp8(w: torch.Tensor):
    _require_cuda(w)
    w = w.contiguous()
    n, k = w.shape
    wq = torch.empty(n, k, dtype=torch.uint8, device=w.device)
    ws = torch.empty(n, dtype=torch.float32, device=w.device)
    check(lib().xn_mm_quantize_weights_fp8(wq.data_ptr(), ws.data_ptr(), w.data_ptr(), _dtype_code(w), n, k, _stream()))
    return wq, ws


def split_rows_e4m3(x: torch.Tensor, want_lo: bool = True):
    return _host.split_rows_e4m3(x, want_lo)


def linear_fp8(x: torch.Tensor, wq: torch.Tensor, w_scale: torch.Tensor, variant: int = 0,
               workspace: torch.Tensor | None = None, out: torch.Tensor | None = None) -> torch.Tensor:
    """y bf16 [m,n] = fp8 linear of bf16 x [m,k]; variant 0 = W8A16, 1 = W8A8."""
    if x.dim() != 2:
        raise XnError(_lib.ERR_INVALID, f"linear_fp8 expects a matrix of activations, got {list(x.shape)}")
    return _host.linear_fp8(x, wq, w_scale, variant, workspace, out)


class LinearFp8:
    """fp8-e4m3 per-channel linear: forward(x bf16) -> bf16."""

    def __init__(self, wq: torch.Tensor, w_scale: torch.Tensor, variant: int = 0):
        self.wq, self.ws, self.variant = wq, w_scale, variant

    @classmethod
    def from_weight(cls, w: torch.Tensor, variant: int = 0) -> "LinearFp8":
        q, s = quantize_weights_fp8(w)
        return cls(q, s, variant)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return _host.linear_fp8(x, self.wq, self.ws, self.variant, None, None)

    __call__ = forward


# ---------------------------------------------------------------------------------------------
# Convolutions: Tensor::conv1d / Tensor::conv_transpose1d (xn-core/src/ops.rs:253-300, 305-350),
# same arguments, same shape rules and error texts; bias fused.
# ---------------------------------------------------------------------------------------------
def conv1d(x: torch.Tensor, kernel: torch.Tensor, bias: torch.Tensor | None = None, stride: int = 1,
           padding: int = 0, dilation: int = 1, groups: int = 1) -> torch.Tensor:
    return _host.conv1d(x, kernel, bias, stride, padding, dilation, groups)


def conv_transpose1d(x: torch.Tensor, kernel: torch.Tensor, bias: torch.Tensor | None = None, stride: int = 1,
                     padding: int = 0, output_padding: int = 0, groups: int = 1) -> torch.Tensor:
    return _host.conv_transpose1d(x, kernel, bias, stride, padding, output_padding, groups)


# ---------------------------------------------------------------------------------------------
# Row operations of a decoder step (xn_mm_rms_norm & co.).
# ---------------------------------------------------------------------------------------------
def rms_norm(x: torch.Tensor, alpha: torch.Tensor, eps: float) -> torch.Tensor:
    return _host.rms_norm(x, alpha, eps)


def softmax(x: torch.Tensor) -> torch.Tensor:
    return _host.softmax(x)


def silu_mul(x: torch.Tensor) -> torch.Tensor:
    return _host.silu_mul(x)


def add(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    return _host.add(a, b)
