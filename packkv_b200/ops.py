"""Device-tensor wrappers over the C ABI (include/packkv_sm100.h).

Everything here takes CUDA tensors, launches on torch's current stream and returns without
synchronising.  Tensors are only the carrier for device memory; the arithmetic is in
libpackkv_sm100.so.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass
from typing import Optional, Tuple

import math

import torch

from . import _lib

HB = {"k": 128, "v": 64}


def _stream_ptr() -> int:
    return torch.cuda.current_stream().cuda_stream


def _require_cuda(*tensors):
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise ValueError("expected CUDA tensors; this library has no CPU path")


def k_block_bound(cb: int, bits: int) -> int:
    lb = 3 if bits >= 4 else 2
    r = cb // 16
    return 2 * r + r * (bits * 16 + lb * 16 + 128 * 2 * bits)


def v_block_bound(cb: int, bits: int) -> int:
    lb = 3 if bits >= 4 else 2
    rpw = 2 if cb == 128 else 1
    ppt = 2 if cb == 32 else 4
    nseg = 2 * rpw
    return 2 * nseg + nseg * (bits * ppt * 4 + lb * ppt * 4 + 32 * ppt * 2 * bits)


def block_bound(which: str, cb: int, bits: int) -> int:
    return k_block_bound(cb, bits) if which == "k" else v_block_bound(cb, bits)


def new_flags(device) -> torch.Tensor:
    return torch.zeros(1, dtype=torch.int32, device=device)


def encode_codes(which: str, codes: torch.Tensor, cb: int, bits: int, *, stream: Optional[torch.Tensor] = None,
                 info: Optional[torch.Tensor] = None, stream_bytes: Optional[torch.Tensor] = None,
                 flags: Optional[torch.Tensor] = None, first_cb: int = 0
                 ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """Bit-packs uint8 codes (n_seq, ctx, hidden) into per-sequence streams.

    Returns (stream (n_seq, capacity) u8, info (n_seq, n_blocks, 2) i32 holding u32 values,
    stream_bytes (n_seq,) i32, flags (1,) i32).  Passing the buffers of an earlier call with
    first_cb > 0 appends the new token blocks behind the existing ones.
    """
    _require_cuda(codes, stream, info, stream_bytes, flags)
    if codes.dtype != torch.uint8 or codes.dim() != 3 or not codes.is_contiguous():
        raise ValueError("codes must be a contiguous uint8 tensor (n_seq, ctx, hidden)")
    n_seq, ctx, hidden = codes.shape
    hb = HB[which]
    if cb <= 0 or ctx % cb or hidden % hb:
        raise ValueError("ctx must be a multiple of cb and hidden a multiple of the block width")
    nhid = hidden // hb
    nblk_new = (ctx // cb) * nhid
    dev = codes.device
    if info is None:
        info = torch.zeros(n_seq, first_cb * nhid + nblk_new, 2, dtype=torch.int32, device=dev)
    if stream is None:
        cap = (first_cb * nhid + nblk_new) * block_bound(which, cb, bits)
        stream = torch.zeros(n_seq, max(16, cap), dtype=torch.uint8, device=dev)
    if stream_bytes is None:
        stream_bytes = torch.zeros(n_seq, dtype=torch.int32, device=dev)
    if flags is None:
        flags = new_flags(dev)
    if info.shape[1] < first_cb * nhid + nblk_new:
        raise ValueError("block_info is too small for the appended blocks")
    fn = _lib.lib().pkv_k_encode if which == "k" else _lib.lib().pkv_v_encode
    st = fn(codes.data_ptr(), codes.stride(0), stream.data_ptr(), stream.stride(0), stream.shape[1],
            info.data_ptr(), info.shape[1], stream_bytes.data_ptr(), flags.data_ptr(),
            n_seq, ctx, hidden, cb, hb, bits, first_cb, _stream_ptr())
    _lib.check(st, f"{which}_encode")
    return stream, info, stream_bytes, flags


def decode_codes(which: str, stream: torch.Tensor, info: torch.Tensor, ctx: int, hidden: int, cb: int, bits: int, *,
                 valid_bytes: Optional[int] = None, flags: Optional[torch.Tensor] = None, first_cb: int = 0,
                 out: Optional[torch.Tensor] = None) -> Tuple[torch.Tensor, torch.Tensor]:
    """Unpacks per-sequence streams back to uint8 codes (n_seq, ctx, hidden)."""
    _require_cuda(stream, info, flags, out)
    if stream.dtype != torch.uint8 or stream.dim() != 2 or stream.stride(1) != 1:
        raise ValueError("stream must be a uint8 tensor (n_seq, capacity)")
    n_seq = stream.shape[0]
    hb = HB[which]
    if out is None:
        out = torch.zeros(n_seq, ctx, hidden, dtype=torch.uint8, device=stream.device)
    if flags is None:
        flags = new_flags(stream.device)
    fn = _lib.lib().pkv_k_decode if which == "k" else _lib.lib().pkv_v_decode
    st = fn(stream.data_ptr(), stream.stride(0), stream.shape[1] if valid_bytes is None else valid_bytes,
            info.data_ptr(), info.shape[1], out.data_ptr(), out.stride(0), flags.data_ptr(),
            n_seq, ctx, hidden, cb, hb, bits, first_cb, _stream_ptr())
    _lib.check(st, f"{which}_decode")
    return out, flags


K_CHANNEL, K_TOKEN, Q_VECTOR, Q_BLOCK = 0, 1, 2, 3


def _param_extents(scale: torch.Tensor, mode: int):
    """(capacity in blocks, capacity in tokens) of a parameter tensor of the given mode; the extent the mode does not
    use is 0."""
    if mode == K_CHANNEL:
        return scale.shape[2], 0
    if mode == K_TOKEN:
        return 0, scale.shape[1]
    if mode == Q_VECTOR:
        return 0, scale.shape[2]
    return scale.shape[1], 0


@dataclass
class Quantised:
    codes: torch.Tensor     # (B, S, H*128) uint8, the encoders' input layout
    scale: torch.Tensor     # channel: (B, H, capacity_blocks, 128); token: (B, capacity_tokens); vector: (B, H, capacity_tokens);
                            # block: (B, capacity_blocks)
    zero: torch.Tensor


def quantize(x: torch.Tensor, block: int, rel: float, mode, *, bits: int = 0, high_precision_zero: bool = False,
             flags: Optional[torch.Tensor] = None, capacity_tokens: Optional[int] = None,
             scale: Optional[torch.Tensor] = None, zero: Optional[torch.Tensor] = None, first_token: int = 0
             ) -> Quantised:
    """Block-quantises x (B, H, S, 128) fp16/bf16 like the reference's quant_ints.

    `mode` is a QuantMode or one of the integers K_CHANNEL / K_TOKEN / Q_VECTOR / Q_BLOCK (the last two are not
    taken by the encoder's single pass or the attention kernel: their codes go through encode_codes).
    Passing existing scale/zero tensors with first_token > 0 writes the new parameters behind
    the ones already there (append path).
    """
    _require_cuda(x, flags, scale, zero)
    if x.dim() != 4 or x.shape[3] != 128 or x.stride(3) != 1 or x.dtype not in (torch.float16, torch.bfloat16):
        raise ValueError("x must be (B, H, S, 128) fp16/bf16 with contiguous channels")
    m = getattr(mode, "value", mode)
    m = {"ChannelQuant": K_CHANNEL, "TokenQuant": K_TOKEN, "VectorQuant": Q_VECTOR, "BlockQuant": Q_BLOCK}.get(m, m)
    if m not in (K_CHANNEL, K_TOKEN, Q_VECTOR, Q_BLOCK):
        raise RuntimeError("not supported")
    B, H, S, D = x.shape
    if S % block:
        raise ValueError("Tensor shape is not divisible by block size")
    cap = max(S + first_token, capacity_tokens or 0)
    dev = x.device
    if flags is None:
        flags = new_flags(dev)
    codes = torch.empty(B, S, H * D, dtype=torch.uint8, device=dev)
    if scale is None:
        shape = {K_CHANNEL: (B, H, cap // block, D), K_TOKEN: (B, cap), Q_VECTOR: (B, H, cap), Q_BLOCK: (B, cap // block)}[m]
        scale = torch.zeros(shape, dtype=x.dtype, device=dev)
        zero = torch.zeros(shape, dtype=x.dtype, device=dev)
    pb, pt = _param_extents(scale, m)
    st = _lib.lib().pkv_quantize(x.data_ptr(), x.stride(0), x.stride(1), x.stride(2), codes.data_ptr(), codes.stride(0),
                                 scale.data_ptr(), zero.data_ptr(), pb, first_token // block, pt, first_token,
                                 B, H, S, block, float(rel), bits, m, int(high_precision_zero),
                                 int(x.dtype == torch.bfloat16), flags.data_ptr(), _stream_ptr())
    _lib.check(st, "quantize")
    return Quantised(codes, scale, zero)


@dataclass
class CompressedLayer:
    """Device-resident compressed KV of one layer: per-sequence K and V streams with their
    block tables and quantisation parameters (layouts: include/packkv_sm100.h)."""
    k_stream: torch.Tensor      # (B, capacity) u8
    k_info: torch.Tensor        # (B, n_k_blocks, 2) i32 (u32 values)
    k_bytes: torch.Tensor       # (B,) i32
    k_scale: torch.Tensor       # channel: (B, Hkv, n_comp/cbk, 128); token: (B, n_comp)
    k_zero: torch.Tensor
    v_stream: torch.Tensor
    v_info: torch.Tensor
    v_bytes: torch.Tensor
    v_scale: torch.Tensor       # (B, n_comp)
    v_zero: torch.Tensor
    n_comp: int
    kv_heads: int
    cbk: int
    cbv: int
    bits_k: int
    bits_v: int
    k_mode: int
    high_precision_zero: bool = False
    order: Optional[torch.Tensor] = None   # (B, n_comp/block, block) u8 when tokens were reordered inside blocks

    def stream_bytes(self) -> int:
        """Compressed payload actually read by a decode step (streams + block tables + scales)."""
        n = int(self.k_bytes.sum().item()) + int(self.v_bytes.sum().item())
        n += self.k_info.numel() * 4 + self.v_info.numel() * 4
        for t in (self.k_scale, self.k_zero, self.v_scale, self.v_zero):
            n += t.numel() * t.element_size()
        return n


def _check_layer_shapes(L: "CompressedLayer", batch: int) -> None:
    """Bounds of everything the attention kernel indexes from n_comp, kv_heads and the block sizes, for layers that are
    read from blobs (serialize.py); a launch checks the same in csrc/host.cpp."""
    if L.cbk not in (64, 128) or L.cbv not in (64, 128) or L.n_comp <= 0 or L.kv_heads <= 0:
        raise RuntimeError("not supported") if L.cbk == 32 or L.cbv == 32 else ValueError("bad layer metadata")
    nkb, nvb = (L.n_comp // L.cbk) * L.kv_heads, (L.n_comp // L.cbv) * 2 * L.kv_heads
    for name in ("k_stream", "v_stream", "k_info", "v_info", "k_scale", "k_zero", "v_scale", "v_zero"):
        t = getattr(L, name)
        if t.shape[0] != batch:
            raise ValueError(f"{name} holds {t.shape[0]} sequences, q holds {batch}")
    if L.k_info.dim() != 3 or L.k_info.shape[2] != 2 or L.k_info.shape[1] < nkb or not L.k_info.is_contiguous():
        raise ValueError(f"k_info must be a contiguous (B, >= {nkb}, 2) table")
    if L.v_info.dim() != 3 or L.v_info.shape[2] != 2 or L.v_info.shape[1] < nvb or not L.v_info.is_contiguous():
        raise ValueError(f"v_info must be a contiguous (B, >= {nvb}, 2) table")
    if L.v_scale.dim() != 2 or L.v_scale.shape[1] < L.n_comp or L.v_zero.shape != L.v_scale.shape:
        raise ValueError("v_scale / v_zero must be (B, >= n_comp)")
    if L.k_mode == K_CHANNEL:
        want = (batch, L.kv_heads)
        if L.k_scale.dim() != 4 or tuple(L.k_scale.shape[:2]) != want or L.k_scale.shape[2] < L.n_comp // L.cbk or L.k_scale.shape[3] != 128 \
                or L.k_zero.shape != L.k_scale.shape:
            raise ValueError("channel-mode k_scale / k_zero must be (B, kv_heads, >= n_comp / cbk, 128)")
    elif L.k_scale.dim() != 2 or L.k_scale.shape[1] < L.n_comp or L.k_zero.shape != L.k_scale.shape:
        raise ValueError("token-mode k_scale / k_zero must be (B, >= n_comp)")
    if L.k_stream.dim() != 2 or L.v_stream.dim() != 2 or L.k_stream.stride(1) != 1 or L.v_stream.stride(1) != 1:
        raise ValueError("streams must be (B, capacity) with contiguous bytes")
    if L.order is not None:
        _check_order(L, batch)


def _check_order(L: "CompressedLayer", batch: int) -> None:
    """One byte for every packed token.  The values are looked at on the device (dense.cu): reading them here would synchronise."""
    order, shape = L.order, L.order.shape
    if order.dtype is not torch.uint8 or len(shape) != 3 or shape[0] != batch or shape[1] * shape[2] != L.n_comp or not order.is_contiguous():
        raise ValueError("order must be a contiguous (B, n_comp / block, block) uint8 tensor")


# changes whenever the attention kernel changes in a way that can change its DRAM traffic (keys recorded profiler figures)
ATTN_KERNEL_REVISION = 3


def decode_attention(q: torch.Tensor, layer: Optional[CompressedLayer], k_res: Optional[torch.Tensor],
                     v_res: Optional[torch.Tensor], n_res: int, *, scaling: Optional[float] = None,
                     out: Optional[torch.Tensor] = None,
                     flags: Optional[torch.Tensor] = None, kv_heads: Optional[int] = None,
                     exchange: Optional["_lib.AttnExchange"] = None, append: Optional[tuple] = None,
                     scratch: Optional[torch.Tensor] = None, plan: Optional[tuple] = None, plan_only: bool = False):
    """softmax(q K^T * scaling) V for one query token per sequence.

    q: (B, Hq, 128) fp16/bf16 (post-RoPE).  `layer` holds the compressed tokens, k_res/v_res
    (B, Hkv, R_cap, 128) the uncompressed residual whose first n_res tokens are valid.
    Returns out (B, Hq, 128) in q's dtype; asynchronous on the current stream.  `exchange` (KV-head-sharded
    decode on several GPUs, see parallel.HeadExchange) makes the launch also deliver the rows to every rank.
    `append` = (k_new, v_new, cos, sin) with k_new / v_new (B, Hkv, 1, 128) and cos / sin (B or 1, 1, 128) or None:
    the launch writes the step's new token (K rotated like rope()) into residual row n_res - 1 before attending;
    n_res counts that token.
    `scratch` (new_attention_scratch) lets the library split a launch with few (sequence, KV head) pairs over
    several clusters per pair in two launches; `plan` = (cluster, nsplit, launches[, extra]), 0 = choose, forces the split
    (extra > 0 with cluster 1: the first `extra` pairs get nsplit + 1 CTAs).
    plan_only: nothing is launched and the plan (cluster, nsplit, launches, extra) that would be used is returned.
    """
    return _lib.host().decode_attention(q, layer, k_res, v_res, n_res, scaling, out, flags, kv_heads, None if exchange is None else ctypes.addressof(exchange),
                                        append, scratch, plan, plan_only)


def decode_attention_narrow(q: torch.Tensor, layer: Optional[CompressedLayer], k_res: Optional[torch.Tensor], v_res: Optional[torch.Tensor], n_res: int, *,
                            scaling: Optional[float], flags: Optional[torch.Tensor] = None, kv_heads: Optional[int] = None, append: Optional[tuple] = None,
                            scratch: Optional[torch.Tensor] = None) -> torch.Tensor:
    """decode_attention for heads of D channels, 64 <= D < 128, a multiple of 8, whose stored rows are widened (widen_rows): q (B, Hq, D)
    from a 16-byte aligned address; the appended rows (B, Hkv, 1, D) and cos / sin (B or 1, 1, D) are widened as they are written.  scaling: the
    factor of the scores, None for 1 / sqrt(D).
    Returns (B, Hq, 128): the first D channels of a row are the head's."""
    return _lib.host().decode_attention_narrow(q, layer, k_res, v_res, n_res, scaling, flags, kv_heads, append, scratch)


def new_attention_scratch(device, nbytes: int = 32 << 20) -> torch.Tensor:
    """Zeroed scratch for decode_attention's two-launch form (scores, per-CTA maxima and sums, per-cluster rows and
    arrival counters); launches that share one must be ordered on one stream."""
    return torch.zeros(nbytes, dtype=torch.uint8, device=device)


def exchange_wait(arrivals: torch.Tensor, n_ranks: int, expected: int, flags: torch.Tensor, max_polls: int = 2_000_000,
                  consume: bool = False) -> None:
    """Makes the current stream wait until this rank's n_ranks arrival counters have reached `expected`
    (modulo 2^32); after max_polls polls (a quarter of a microsecond apart) the wait gives up and sets FLAG_TIMEOUT.
    consume: `expected` is the arrivals of one step and is taken off the counters again once they are all there, so
    that the same call serves every step (CUDA graphs)."""
    _require_cuda(arrivals, flags)
    fn = _lib.lib().pkv_exchange_wait_consume if consume else _lib.lib().pkv_exchange_wait
    st = fn(arrivals.data_ptr(), n_ranks, expected & 0xFFFFFFFF, max_polls, flags.data_ptr(), _stream_ptr())
    _lib.check(st, "exchange_wait")


def rope(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """(x * cos) + (rotate_half(x) * sin) with the reference's per-op rounding.
    x (B, H, T, D) with contiguous channels; cos/sin (B or 1, T, D)."""
    return _lib.host().rope(x, cos, sin, out)


def append_residual(k_new: torch.Tensor, v_new: torch.Tensor, k_res: torch.Tensor, v_res: torch.Tensor, position: int,
                    cos: Optional[torch.Tensor] = None, sin: Optional[torch.Tensor] = None) -> None:
    """Writes the new tokens (B, H, T, 128) into rows [position, position+T) of the residual buffers
    (B, H, capacity, 128): K after RoPE (skipped when cos/sin are None), V as is.  One launch."""
    _lib.host().append_residual(k_new, v_new, k_res, v_res, position, cos, sin)


def waiting_step(k_res: torch.Tensor, k_new: torch.Tensor, v_new: torch.Tensor, cos: Optional[torch.Tensor], sin: Optional[torch.Tensor]) -> Optional[int]:
    """The current stream (its handle) if decode_attention(append=(k_new, v_new, cos, sin)) over residual buffers like k_res can take these
    tensors as they are; None if they have to be converted, or refused, first."""
    return _lib.host().waiting_step(k_res, k_new, v_new, cos, sin)


def stream_of(t: torch.Tensor) -> int:
    """Handle of the current stream of t's device (torch.cuda.current_stream(t.device).cuda_stream, without building the Python objects)."""
    return _lib.host().stream_of(t)


def widen_rows(k: torch.Tensor, v: Optional[torch.Tensor], k_out: torch.Tensor, v_out: Optional[torch.Tensor], position: int = 0,
               cos: Optional[torch.Tensor] = None, sin: Optional[torch.Tensor] = None, zero_tail: bool = False) -> None:
    """append_residual for heads of 64 <= D < 128 channels (B, H, T, D): the rows of k_out / v_out (B, H, capacity, 128) are
    widened, channels D.. repeating the row's first 128 - D (zeros with zero_tail).  v and v_out may be None.  One launch."""
    _lib.host().widen_rows(k, v, k_out, v_out, position, cos, sin, zero_tail)


def dequantize(codes: torch.Tensor, scale: torch.Tensor, zero: torch.Tensor, heads: int, block: int, mode: int, *,
               first_token: int = 0, high_precision_zero: bool = False, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """codes (B, T, heads*128) uint8 + scale/zero -> dense (B, heads, T, 128) in scale's dtype."""
    _require_cuda(codes, scale, zero, out)
    B, T, _ = codes.shape
    if out is None:
        out = torch.empty(B, heads, T, 128, dtype=scale.dtype, device=codes.device)
    pb, pt = _param_extents(scale, mode)
    st = _lib.lib().pkv_dequantize(codes.data_ptr(), codes.stride(0), scale.data_ptr(), zero.data_ptr(), pb, pt, first_token,
                                   out.data_ptr(), out.stride(0), out.stride(1), out.stride(2), B, heads, T, block, mode,
                                   int(high_precision_zero), int(scale.dtype == torch.bfloat16), _stream_ptr())
    _lib.check(st, "dequantize")
    return out


def dense(which: str, layer: CompressedLayer, res: Optional[torch.Tensor], n_res: int, dim: int, block: int,
          flags: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Rows of K or V of a layer as the reference's cache returns them, (B, H, n_comp + n_res, dim): the packed tokens
    dequantised (in source order when the layer is reordered) and the first n_res rows of the residual behind them.
    `block` is the quantisation block; dim < 128 keeps the first channels of every head.  One launch."""
    get = lambda name: getattr(layer, f"{which}_{name}")
    stream, info, scale, zero = get("stream"), get("info"), get("scale"), get("zero")
    B, H, n, cb = stream.shape[0], layer.kv_heads, layer.n_comp, layer.cbk if which == "k" else layer.cbv
    mode = layer.k_mode if which == "k" else K_TOKEN
    _require_cuda(stream, info, scale, zero, res, layer.order, flags)
    if flags is None:
        flags = new_flags(stream.device)
    pb, pt = _param_extents(scale, mode)
    if (mode == K_CHANNEL and n % block) or n % cb or info.dim() != 3 or info.shape[1] < (n // cb) * H * (1 if which == "k" else 2) or not info.is_contiguous() \
            or stream.dim() != 2 or stream.stride(1) != 1 or (pb < n // block if mode == K_CHANNEL else pt < n) \
            or not scale.is_contiguous() or not zero.is_contiguous() or zero.shape != scale.shape or info.shape[0] != B or scale.shape[0] != B:
        raise ValueError("dense: the layer's tables do not cover its tokens")
    order_block = block
    if layer.order is not None:
        _check_order(layer, B)
        order_block = layer.order.shape[2]
    if n_res and (res.dim() != 4 or res.shape[:2] != (B, H) or res.shape[2] < n_res or res.shape[3] != 128 or res.stride(3) != 1 or res.stride(2) != 128
                  or res.dtype != scale.dtype):
        raise ValueError("dense: the residual must be (B, H, >= n_res, 128) rows of the layer's element type")
    out = torch.empty(B, H, n + n_res, dim, dtype=scale.dtype, device=scale.device)
    a = _lib.DenseArgs(stream.data_ptr(), stream.stride(0), stream.shape[1], info.data_ptr(), info.shape[1], scale.data_ptr(), zero.data_ptr(), pb, pt,
                       None if layer.order is None else layer.order.data_ptr(), n, res.data_ptr() if n_res else None,
                       res.stride(0) if n_res else 0, res.stride(1) if n_res else 0, out.data_ptr(), out.stride(0), out.stride(1), out.stride(2),
                       flags.data_ptr(), B, H, dim, n, n_res, order_block, block, cb, 0 if which == "k" else 1,
                       layer.bits_k if which == "k" else layer.bits_v, mode, int(layer.high_precision_zero), int(scale.dtype == torch.bfloat16))
    _lib.check(_lib.lib().pkv_dense(ctypes.byref(a), _stream_ptr()), "dense")
    return out


def encode_tensor(which: str, x: torch.Tensor, block: int, rel: float, mode: int, bits: int, cb: int, *,
                  scale: torch.Tensor, zero: torch.Tensor, stream: torch.Tensor, info: torch.Tensor,
                  stream_bytes: torch.Tensor, flags: torch.Tensor, first_token: int = 0,
                  high_precision_zero: bool = False, scratch: Optional[torch.Tensor] = None,
                  order: Optional[torch.Tensor] = None, order_block: int = 64) -> None:
    """Quantises x (B, H, S, 128) and packs it behind the `first_token` tokens already in the
    streams (one C call).  `scratch` (uint8, >= B*S*H*128 bytes) holds the codes in between; one is
    allocated when not given.  `order` (B, S/order_block, order_block) uint8 (value_median_order): rows are read
    through it, i.e. the tokens of every reorder block are stored in that order (single-pass modes only:
    RuntimeError("not supported") otherwise)."""
    _lib.host().encode_tensor(which, x, block, rel, mode, bits, cb, scale, zero, stream, info, stream_bytes, flags, first_token, high_precision_zero,
                              scratch, order, order_block)


def value_median_order(v: torch.Tensor, block: int, rel: float, flags: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Token order of every block by descending lower median of the V codes (stable on ties), computed from
    fp16/bf16 V (B, H <= 8, S, 128) without a code matrix: the same order as median_order on quantised codes.
    Returns (B, S/block, block) uint8."""
    return _lib.host().value_median_order(v, block, rel, flags)


def encode_tensor_static(which: str, x: torch.Tensor, block: int, rel: float, mode: int, bits: int, cb: int, *,
                         scale: torch.Tensor, zero: torch.Tensor, stream: torch.Tensor, info: torch.Tensor,
                         stream_bytes: torch.Tensor, flags: torch.Tensor, first_token: int = 0,
                         high_precision_zero: bool = False) -> None:
    """encode_tensor for callers that must stay away from the device allocator (a serving engine's
    decode loop whose memory pool owns all free HBM: an allocation there can fail or stall the
    device).  The codes go through a 16 MiB array built into the library, so B*S*H*128 must not
    exceed that (ValueError otherwise), and calls must not overlap on the GPU because they share
    it.  The first call on a device resolves the array's address: make it before capturing streams.
    Results are identical to encode_tensor's."""
    _lib.host().encode_tensor(which, x, block, rel, mode, bits, cb, scale, zero, stream, info, stream_bytes, flags, first_token, high_precision_zero,
                              False, None, 0)


def median_order(v_codes: torch.Tensor, heads: int, block: int, want_keys: bool = False):
    """Token order of every block by descending lower-median of the V codes (stable on ties).
    v_codes (B, S, heads*128) uint8 -> order (B, S/block, block) uint8 [, keys (B, S) uint8]."""
    _require_cuda(v_codes)
    B, S, _ = v_codes.shape
    order = torch.empty(B, S // block, block, dtype=torch.uint8, device=v_codes.device)
    keys = torch.empty(B, S, dtype=torch.uint8, device=v_codes.device) if want_keys else None
    st = _lib.lib().pkv_median_order(v_codes.data_ptr(), v_codes.stride(0), order.data_ptr(),
                                     keys.data_ptr() if want_keys else None, B, heads, S, block, _stream_ptr())
    _lib.check(st, "median_order")
    return (order, keys) if want_keys else order


def greedy_order(k_codes: torch.Tensor, v_codes: torch.Tensor, heads: int, block: int, pack_len: int = 16) -> torch.Tensor:
    """Token order of every block by the reference's greedy repacking heuristic
    (utils/compute.py:210-260) on the K||V code vectors of each token.
    k_codes, v_codes (B, S, heads*128) uint8 -> order (B, S/block, block) uint8."""
    _require_cuda(k_codes, v_codes)
    if k_codes.shape != v_codes.shape or k_codes.stride() != v_codes.stride():
        raise ValueError("k_codes and v_codes must have the same shape and strides")
    B, S, _ = k_codes.shape
    order = torch.empty(B, S // block, block, dtype=torch.uint8, device=k_codes.device)
    st = _lib.lib().pkv_greedy_order(k_codes.data_ptr(), v_codes.data_ptr(), k_codes.stride(0), order.data_ptr(),
                                     B, heads, S, block, pack_len, _stream_ptr())
    _lib.check(st, "greedy_order")
    return order


def size_model(codes: torch.Tensor, pack_len: int = 16) -> int:
    """Bytes the reference's bit_pack estimate (utils/compute.py:272-297) gives for one code tensor
    (B, S, hidden) uint8 (synchronises to read the two counters back)."""
    _require_cuda(codes)
    B, S, hidden = codes.shape
    bits = torch.zeros(1, dtype=torch.int64, device=codes.device)
    present = torch.zeros(8, dtype=torch.int32, device=codes.device)
    st = _lib.lib().pkv_size_model(codes.data_ptr(), codes.stride(0), B, S, hidden, pack_len, bits.data_ptr(), present.data_ptr(), _stream_ptr())
    _lib.check(st, "size_model")
    n_values = sum(bin(int(w) & 0xFFFFFFFF).count("1") for w in present.tolist())
    if n_values == 0:
        return 0
    b = math.ceil(math.log2(n_values))
    n_packs = B * (S // pack_len) * hidden
    return (int(bits.item()) * pack_len + n_packs * (b + math.ceil(math.log2(b + 1)))) // 8


def gather_rows(codes: torch.Tensor, order: torch.Tensor, block: int) -> torch.Tensor:
    """Applies `order` to the token rows of a code matrix (B, S, row_bytes)."""
    _require_cuda(codes, order)
    B, S, rb = codes.shape
    out = torch.empty_like(codes)
    st = _lib.lib().pkv_gather_rows(codes.data_ptr(), out.data_ptr(), codes.stride(0), order.data_ptr(), B, S, block, rb, _stream_ptr())
    _lib.check(st, "gather_rows")
    return out


def gather_params(params: torch.Tensor, order: torch.Tensor, block: int, tokens: int, first: int = 0) -> torch.Tensor:
    """Applies `order` to per-token parameters (B, row_len) for tokens [first, first+tokens)."""
    _require_cuda(params, order)
    out = params.clone()
    st = _lib.lib().pkv_gather_params(params.data_ptr(), out.data_ptr(), params.shape[1], first, order.data_ptr(),
                                      params.shape[0], tokens, block, _stream_ptr())
    _lib.check(st, "gather_params")
    return out
