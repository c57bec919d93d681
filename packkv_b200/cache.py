"""KV-cache classes with the reference's names and call contract
(models/cache/packkv_cache.py:22-38, models/cache/packkv_quant.py:9-130), backed by the
compressed store instead of a quantise->dequantise simulation.

    PackKVCacheConfigStatic.config = PackKVCacheConfig(...)
    cache = PackKVCache(batch_size, head_num, head_dim, layer_num)
    k_all, v_all = cache.update(key_states, value_states, layer_idx, {"cos": cos, "sin": sin})
    out = cache.attend(query_states, layer_idx)          # fused decompress-attention (decode)

`update` applies RoPE to K inside the cache, appends to the uncompressed residual, and moves whole
token blocks into the packed streams by the reference's cut rule (utils/compute.py:54-67): with
block 64 and buffer 192 the residual holds 128..191 tokens and every 64th decode step packs one
block.  For prefill (more than one new token), for `materialize=True` and when quantisation is
disabled it returns dense K/V exactly like the reference (dequantised history + residual); on a
decode step with `materialize=False` it returns (None, None) and `attend` computes the attention
straight from the packed streams.

With the installed transformers (5.x) the attention modules rotate K themselves and call
`update(key_states, value_states, layer_idx)` without sin/cos: then no RoPE is applied here.
`decode_handles=True` makes a decode step return a pair of `PackKVHandle`s instead of
(None, None); the attention function registered by `packkv_b200.hf` turns them into a call of
`attend`.
"""
from __future__ import annotations

import math
from typing import Any, Dict, List, Optional, Tuple

import torch

from . import encode, ops
from .config import PackKVCacheConfig, QuantMode, RepackMethod

try:  # the installed transformers' Cache needs constructor arguments the reference never passed
    from transformers import Cache as _HFCache
except Exception:  # pragma: no cover - transformers is optional
    _HFCache = object


class PackKVCacheConfigStatic:
    """Process-wide configuration slot, as in the reference (packkv_quant.py:9-11)."""
    config: Optional[PackKVCacheConfig] = None
    extract_cache = None


def bits_for_rel(rel: float) -> int:
    """Bit width the quantiser's codes need: it produces at most round(1/rel) + 2 levels."""
    return max(2, math.ceil(math.log2(math.floor(1.0 / rel + 1e-6) + 2)))


def compress_block_count(length: int, block: int, recent: int) -> int:
    """Whole blocks that leave a residual of `length` tokens (utils/compute.py:60-62)."""
    return max(0, (length + block - length % block - recent) // block)


def _zeroed(device, **specs) -> Dict[str, torch.Tensor]:
    """Zeroed tensors, name=(shape, dtype), in one allocation that one launch clears: the ten tensors of a layer took ten launches (two layers
    of 4 x 8191 tokens: 638 us with them, 592 without).  Each starts on a 256-byte boundary, as an allocation of its own would at least."""
    sizes = {name: math.prod(shape) * dtype.itemsize for name, (shape, dtype) in specs.items()}
    store = torch.zeros(sum((n + 255) // 256 * 256 for n in sizes.values()), dtype=torch.uint8, device=device)
    out, at = {}, 0
    for name, (shape, dtype) in specs.items():
        out[name] = store[at: at + sizes[name]].view(dtype).view(shape)
        at += (sizes[name] + 255) // 256 * 256
    return out


class PackKVHandle:
    """Stands in for the K (or V) tensor of a decode step: names the cache and the layer."""
    __slots__ = ("cache", "layer_idx")

    def __init__(self, cache: "PackKVCache", layer_idx: int):
        self.cache, self.layer_idx = cache, layer_idx


class _Layer:
    def __init__(self):
        self.comp: Optional[ops.CompressedLayer] = None
        self.capacity = 0          # tokens the compressed store has room for
        self.k_res: Optional[torch.Tensor] = None
        self.v_res: Optional[torch.Tensor] = None
        self.n_res = 0
        self.n_comp = 0
        self.pending = None        # (k_new, v_new, cos, sin) of a decode step whose token the next attend() writes into row n_res - 1
        self.pending_on = 0        # the stream that update() was called on with them


class PackKVCache(_HFCache):
    """Compressed K and V of a model's layers behind the reference's update() / get_seq_length() (packkv_cache.py:22-38).

    The buffers of a layer are the cache's own: a residual that overflows continues in new buffers, and a store that is full
    in a larger one, so an address read from outside is good until the next update()."""

    def __init__(self, batch_size, head_num, head_dim, layer_num, materialize: bool = False, decode_handles: bool = False):
        if _HFCache is not object:
            try:
                super().__init__(layers=[])
            except TypeError:
                try:
                    super().__init__()
                except Exception:
                    pass
        self.batch_size = batch_size
        self.head_num = head_num          # the models pass num_attention_heads; KV heads come from the tensors
        self.head_dim = head_dim
        self.materialize = materialize
        self.decode_handles = decode_handles
        self._layers: List[_Layer] = [_Layer() for _ in range(layer_num)]
        self.flags: Optional[torch.Tensor] = None
        self._scratch: Optional[torch.Tensor] = None   # hand-over area of the attention's two-launch form

    # ---------------------------------------------------------------------------------------------
    @staticmethod
    def _config() -> PackKVCacheConfig:
        cfg = PackKVCacheConfigStatic.config
        if cfg is None:
            raise ValueError("TComCacheConfigStatic.config is not set. Please set it before using TComCache.")
        return cfg

    def check_flags(self):
        """Reads the device status word (synchronises) and raises if a kernel reported a condition that makes
        the cache's contents or an attention result wrong.  update() and attend() are asynchronous and do not
        call this; compressed_bytes() does, and callers should at points where they synchronise anyway."""
        f = int(self.flags.item()) if self.flags is not None else 0
        if f:
            raise RuntimeError(f"PackKV device status flags set: {f} (1=stream overflow, 2=code range, 4=bad stream, "
                               "8=wait timed out, 16=zero-point outside the exact range of the attention kernel)")

    _check_flags = check_flags

    def _ensure_store(self, L: _Layer, kv_heads: int, need_tokens: int, dtype, device, cfg: PackKVCacheConfig):
        if L.comp is not None and L.capacity >= need_tokens:
            return
        block = cfg.block_size
        cap = max(need_tokens, 2 * L.capacity, 16 * block)
        cap = (cap + 127) // 128 * 128
        bits_k, bits_v = bits_for_rel(cfg.k_quant_scale_rel), bits_for_rel(cfg.v_quant_scale_rel)
        k_mode = cfg.quant_method.value[0]
        B = self.batch_size
        k_params = (B, kv_heads, cap // block, 128) if k_mode == QuantMode.ChannelQuant else (B, cap)
        new = ops.CompressedLayer(
            **_zeroed(device,
                      k_stream=((B, encode.stream_capacity("k", cap, kv_heads, block, bits_k)), torch.uint8),
                      k_info=((B, (cap // block) * kv_heads, 2), torch.int32), k_bytes=((B,), torch.int32), k_scale=(k_params, dtype), k_zero=(k_params, dtype),
                      v_stream=((B, encode.stream_capacity("v", cap, kv_heads, block, bits_v)), torch.uint8),
                      v_info=((B, (cap // block) * 2 * kv_heads, 2), torch.int32), v_bytes=((B,), torch.int32), v_scale=((B, cap), dtype), v_zero=((B, cap), dtype)),
            n_comp=0, kv_heads=kv_heads, cbk=block, cbv=block, bits_k=bits_k, bits_v=bits_v,
            k_mode=ops.K_CHANNEL if k_mode == QuantMode.ChannelQuant else ops.K_TOKEN,
            high_precision_zero=bool(cfg.high_precision_zero_point))
        old = L.comp
        if old is not None:   # grow: copy the used prefix of every buffer
            new.k_stream[:, : old.k_stream.shape[1]] = old.k_stream
            new.v_stream[:, : old.v_stream.shape[1]] = old.v_stream
            new.k_info[:, : old.k_info.shape[1]] = old.k_info
            new.v_info[:, : old.v_info.shape[1]] = old.v_info
            new.k_bytes.copy_(old.k_bytes)
            new.v_bytes.copy_(old.v_bytes)
            if new.k_mode == ops.K_CHANNEL:
                new.k_scale[:, :, : old.k_scale.shape[2]] = old.k_scale
                new.k_zero[:, :, : old.k_zero.shape[2]] = old.k_zero
            else:
                new.k_scale[:, : old.k_scale.shape[1]] = old.k_scale
                new.k_zero[:, : old.k_zero.shape[1]] = old.k_zero
            new.v_scale[:, : old.v_scale.shape[1]] = old.v_scale
            new.v_zero[:, : old.v_zero.shape[1]] = old.v_zero
            new.n_comp = old.n_comp
            new.order = old.order
        L.comp, L.capacity = new, cap

    def _compress(self, L: _Layer, k: torch.Tensor, v: torch.Tensor, cfg: PackKVCacheConfig):
        """Quantises and packs k, v (B, H, n*block, 128) behind the tokens already stored."""
        B, H, n, _ = k.shape
        self._ensure_store(L, H, L.n_comp + n, k.dtype, k.device, cfg)
        C, block = L.comp, cfg.block_size
        if self.flags is None:
            self.flags = ops.new_flags(k.device)
        first, order = L.n_comp, None
        if cfg.repack_method == RepackMethod.MEDIAN and encode.median_in_one_pass(k, v, block, C):
            # the order straight from V; the encoders then read their rows through it
            order = ops.value_median_order(v, block, cfg.v_quant_scale_rel, flags=self.flags)
            C.order = order if C.order is None else torch.cat([C.order, order], dim=1)
        if order is None and cfg.repack_method in (RepackMethod.MEDIAN, RepackMethod.GREEDY):
            # quantise, reorder the tokens of each new block (median of the V codes, or greedy packs), pack
            kq = ops.quantize(k, block, cfg.k_quant_scale_rel, C.k_mode, bits=C.bits_k, high_precision_zero=C.high_precision_zero,
                              flags=self.flags, scale=C.k_scale, zero=C.k_zero, first_token=L.n_comp)
            vq = ops.quantize(v, block, cfg.v_quant_scale_rel, ops.K_TOKEN, bits=C.bits_v, high_precision_zero=C.high_precision_zero,
                              flags=self.flags, scale=C.v_scale, zero=C.v_zero, first_token=L.n_comp)
            order = (ops.median_order(vq.codes, H, block) if cfg.repack_method == RepackMethod.MEDIAN
                     else ops.greedy_order(kq.codes, vq.codes, H, block, cfg.pack_size))
            C.v_scale = ops.gather_params(C.v_scale, order, block, n, first=L.n_comp)
            C.v_zero = ops.gather_params(C.v_zero, order, block, n, first=L.n_comp)
            if C.k_mode == ops.K_TOKEN:
                C.k_scale = ops.gather_params(C.k_scale, order, block, n, first=L.n_comp)
                C.k_zero = ops.gather_params(C.k_zero, order, block, n, first=L.n_comp)
            ops.encode_codes("k", ops.gather_rows(kq.codes, order, block), C.cbk, C.bits_k, stream=C.k_stream, info=C.k_info,
                             stream_bytes=C.k_bytes, flags=self.flags, first_cb=L.n_comp // C.cbk)
            ops.encode_codes("v", ops.gather_rows(vq.codes, order, block), C.cbv, C.bits_v, stream=C.v_stream, info=C.v_info,
                             stream_bytes=C.v_bytes, flags=self.flags, first_cb=L.n_comp // C.cbv)
            C.order = order if C.order is None else torch.cat([C.order, order], dim=1)
        else:
            more = dict(flags=self.flags, first_token=first, high_precision_zero=C.high_precision_zero,
                        scratch=torch.empty(max(16, B * n * H * 128), dtype=torch.uint8, device=k.device), order=order, order_block=block)
            ops.encode_tensor("k", k, block, cfg.k_quant_scale_rel, C.k_mode, C.bits_k, C.cbk, scale=C.k_scale, zero=C.k_zero,
                              stream=C.k_stream, info=C.k_info, stream_bytes=C.k_bytes, **more)
            ops.encode_tensor("v", v, block, cfg.v_quant_scale_rel, ops.K_TOKEN, C.bits_v, C.cbv, scale=C.v_scale, zero=C.v_zero,
                              stream=C.v_stream, info=C.v_info, stream_bytes=C.v_bytes, **more)
        L.n_comp += n
        C.n_comp = L.n_comp

    # ---------------------------------------------------------------------------------------------
    def update(self, key_states: torch.Tensor, value_states: torch.Tensor, layer_idx: int,
               cache_kwargs: Optional[Dict[str, Any]] = None, **_unused) -> Tuple[Optional[torch.Tensor], Optional[torch.Tensor]]:
        """Adds T tokens, (B, KV heads, T, D) each, to a layer; the module's description says what is returned.

        A single token of 128 channels is written into the residual by the launch that attends: its tensors, cos and sin among them, must stay
        as they are until this layer's attend(), flush(), dense() or next update() has been called.  Those of every other call (prompts, narrow
        heads, materialize) have been read, in stream order, when update() returns."""
        cfg = self._config()
        if PackKVCacheConfigStatic.extract_cache is not None:
            assert not cfg.enable_quant, "Disable quant to enable cache collect."
        L = self._layers[layer_idx]
        self._flush(L)
        B, H, T, D = key_states.shape
        if D != 128 and (D > 128 or D < 64 or D % 8):
            raise RuntimeError("not supported")   # streams are built from 128-channel blocks; 64..120 are widened, see _append
        if cfg.enable_quant and cfg.block_size not in (64, 128):
            # the codec packs 32-token blocks too, but the attention kernel reads 64- and 128-token blocks only:
            # refuse here, not at the first attend()
            raise RuntimeError("not supported: PackKVCache needs block_size 64 or 128")
        # the reference's models pass K before RoPE together with sin/cos; the installed transformers rotates K itself
        cos, sin = (cache_kwargs["cos"], cache_kwargs["sin"]) if cache_kwargs is not None and "cos" in cache_kwargs and "sin" in cache_kwargs else (None, None)
        if not cfg.enable_quant:
            return self._update_dense(L, key_states, value_states, cos, sin, layer_idx)
        total = L.n_res + T
        n_c = compress_block_count(total, cfg.block_size, cfg.buffer_size) * cfg.block_size
        if n_c == 0 and L.k_res is not None and T == 1 and D == 128 and not self.materialize:
            on = ops.waiting_step(L.k_res, key_states, value_states, cos, sin)
            if on is not None:
                # the common decode step: the fused attention to follow writes the token into the residual itself (attend() below).  What the
                # launch would not take goes through _append at once, which converts it, or refuses it before the token is counted.
                L.pending, L.pending_on = (key_states, value_states, cos, sin), on
                L.n_res = total
                return self._step_result(layer_idx, T)
        if key_states.stride(3) != 1 or value_states.stride(3) != 1:
            key_states, value_states = key_states.contiguous(), value_states.contiguous()
        if value_states.dtype != key_states.dtype:
            value_states = value_states.to(key_states.dtype)
        if L.k_res is None:
            L.k_res = key_states.new_empty(B, H, cfg.buffer_size + cfg.block_size, 128)
            L.v_res = torch.empty_like(L.k_res)

        def part(t, lo, hi):                     # tokens lo..hi of the cos / sin tables
            return None if t is None else t[..., lo:hi, :]

        if n_c == 0:
            self._append(L.k_res, L.v_res, L.n_res, key_states, value_states, cos, sin)
            L.n_res = total
        elif L.n_res == 0:
            # the first tokens: what is packed goes through the rotation (and the widening) once, what stays behind
            # straight into the residual
            if cos is not None and (cos.dim() < 2 or cos.shape[-2] != T or sin.shape != cos.shape):
                raise ValueError("cos/sin must be (B or 1, T, D)")      # parts of longer tables would rotate by other positions
            k_head, v_head = key_states[:, :, :n_c], value_states[:, :, :n_c]
            if D != 128:
                k_wide, v_wide = (key_states.new_empty(B, H, n_c, 128) for _ in range(2))
                self._append(k_wide, v_wide, 0, k_head, v_head, part(cos, 0, n_c), part(sin, 0, n_c))
                k_head, v_head = k_wide, v_wide
            else:
                k_head = ops.rope(k_head, part(cos, 0, n_c), part(sin, 0, n_c)) if cos is not None else k_head.contiguous()
            self._compress(L, k_head, v_head, cfg)
            if total > n_c:
                self._append(L.k_res, L.v_res, 0, key_states[:, :, n_c:], value_states[:, :, n_c:], part(cos, n_c, T), part(sin, n_c, T))
            L.n_res = total - n_c
        else:
            # the residual overflows: its first blocks are packed, the rows behind them start a new one
            k_all, v_all = L.k_res, L.v_res
            if total > k_all.shape[2]:
                k_all = key_states.new_empty(B, H, total, 128)
                v_all = torch.empty_like(k_all)
                self._append(k_all, v_all, 0, L.k_res[:, :, : L.n_res], L.v_res[:, :, : L.n_res], None, None)
            self._append(k_all, v_all, L.n_res, key_states, value_states, cos, sin)
            self._compress(L, k_all[:, :, :n_c], v_all[:, :, :n_c], cfg)
            k_res = torch.empty_like(L.k_res)
            v_res = torch.empty_like(k_res)
            if total > n_c:
                self._append(k_res, v_res, 0, k_all[:, :, n_c:total], v_all[:, :, n_c:total], None, None)
            L.k_res, L.v_res, L.n_res = k_res, v_res, total - n_c
        return self._step_result(layer_idx, T)

    @staticmethod
    def _update_dense(L: "_Layer", key_states, value_states, cos, sin, layer_idx: int):
        """enable_quant off: the cache keeps (and, when asked, collects) the uncompressed K and V."""
        k_new = ops.rope(key_states, cos, sin) if cos is not None else key_states.contiguous()
        v_new = value_states
        L.k_res = k_new if L.k_res is None else torch.cat([L.k_res[:, :, : L.n_res], k_new], dim=2)
        L.v_res = v_new.clone() if L.v_res is None else torch.cat([L.v_res[:, :, : L.n_res], v_new], dim=2)
        L.n_res += key_states.shape[2]
        ex = PackKVCacheConfigStatic.extract_cache
        if ex is not None:
            ex.key_caches.setdefault(0, {})[layer_idx - 1] = L.k_res
            ex.value_caches.setdefault(0, {})[layer_idx - 1] = L.v_res
        return L.k_res, L.v_res

    @staticmethod
    def _append(k_rows: torch.Tensor, v_rows: torch.Tensor, position: int, k: torch.Tensor, v: torch.Tensor, cos, sin) -> None:
        """Tokens (B, H, T, D) into rows [position, position + T) of 128 channels: K rotated when cos is given; rows of
        64 <= D < 128 are widened, the tail repeating the first 128 - D channels.  The streams are built from 128-channel
        blocks; with copies in the tail the per-channel K parameters of the real channels and the per-token minima / maxima
        of V (and token-mode K) are unchanged, so codes and parameters of the real channels are exactly the reference's for
        head_dim D.  attend() pads q with zeros, so the copies add nothing to the scores, and drops the output's tail."""
        if not k.is_cuda or k.dtype not in (torch.float16, torch.bfloat16):
            # kept uncompressed as it is (packing and attention refuse it)
            if cos is not None:
                k = ops.rope(k, cos, sin)
            tail = k_rows.shape[3] - k.shape[3]
            k, v = (torch.cat([t, t[..., :tail]], dim=-1) if tail else t for t in (k, v))
            k_rows[:, :, position: position + k.shape[2]], v_rows[:, :, position: position + k.shape[2]] = k, v
        elif k.shape[3] == 128:
            ops.append_residual(k, v, k_rows, v_rows, position, cos, sin)
        else:
            ops.widen_rows(k, v, k_rows, v_rows, position, cos, sin)

    def _flush(self, L: "_Layer") -> None:
        """Writes a decode step's token that no attend() has consumed into the residual (one launch)."""
        if L.pending is not None:
            k_new, v_new, cos, sin = L.pending
            ops.append_residual(k_new, v_new, L.k_res, L.v_res, L.n_res - 1, cos, sin)
            self._written(L)

    @staticmethod
    def _written(L: "_Layer") -> None:
        """The launch that reads a step's tensors has been made: they are let go.  On another stream than update()'s the allocator is told
        first, or it would give their memory to that stream's next tensors while the launch still waits or reads."""
        if L.pending is not None:
            if ops.stream_of(L.k_res) != L.pending_on:
                for t in L.pending:
                    if t is not None:
                        t.record_stream(torch.cuda.current_stream(L.k_res.device))
            L.pending = None

    def flush(self) -> None:
        """Makes the residual buffers of every layer complete (call before reading them from outside)."""
        for L in self._layers:
            self._flush(L)

    def _step_result(self, layer_idx: int, T: int):
        if T > 1 or self.materialize:
            return self.dense(layer_idx)
        if self.decode_handles:
            return PackKVHandle(self, layer_idx), PackKVHandle(self, layer_idx)
        return None, None

    def dense(self, layer_idx: int) -> Tuple[torch.Tensor, torch.Tensor]:
        """Dequantised history + residual, (B, H, S, 128): what the reference's update returns."""
        L = self._layers[layer_idx]
        self._flush(L)
        D = self.head_dim if self.head_dim < 128 else 128
        if L.n_comp == 0:
            return L.k_res[:, :, : L.n_res, :D].clone(), L.v_res[:, :, : L.n_res, :D].clone()
        if self.flags is None:            # a restored cache that has neither packed a block nor attended yet
            self.flags = ops.new_flags(L.comp.k_stream.device)
        block = self._config().block_size
        return (ops.dense("k", L.comp, L.k_res, L.n_res, D, block, self.flags), ops.dense("v", L.comp, L.v_res, L.n_res, D, block, self.flags))

    def attend(self, query_states: torch.Tensor, layer_idx: int, scaling: Optional[float] = None) -> torch.Tensor:
        """Decode attention for one new token: query_states (B, Hq, 1, 128) after RoPE ->
        (B, 1, Hq, 128), the layout the reference's eager attention returns (llama.py:210-212).  Writes the token that update() left for it;
        a call that raises leaves it in place."""
        L = self._layers[layer_idx]
        B, Hq, T, D = query_states.shape
        if T != 1:
            raise ValueError("attend handles one query token per sequence; use dense() for prefill")
        if self.flags is None:
            self.flags = ops.new_flags(query_states.device)
        q = query_states.reshape(B, Hq, D).contiguous()
        kv_heads = L.comp.kv_heads if L.comp is not None else L.k_res.shape[1]
        if self._scratch is None and B * kv_heads <= 64:
            # few (sequence, KV head) pairs: let the library split each over several clusters (all layers share the
            # area: their launches are ordered on one stream)
            self._scratch = ops.new_attention_scratch(q.device)
        if D != 128:
            self._flush(L)                                     # (of a token of 128 channels; narrow heads' rows are written by update())
            if q.data_ptr() % 16:
                q = q.clone()
            # the launch reads q's D channels as if zeros stood behind them (the copied channels of K add nothing).  It could widen the
            # step's rows too, but update() would then have to keep the caller's tensors instead of their contents until here.
            out = ops.decode_attention_narrow(q, L.comp if L.n_comp else None, L.k_res, L.v_res, L.n_res, scaling=D ** -0.5 if scaling is None else scaling,
                                              flags=self.flags, kv_heads=kv_heads, scratch=self._scratch)
            return out.view(B, 1, Hq, 128)[..., :D]
        out = ops.decode_attention(q, L.comp if L.n_comp else None, L.k_res, L.v_res, L.n_res, scaling=scaling,
                                   flags=self.flags, kv_heads=kv_heads, append=L.pending, scratch=self._scratch)
        self._written(L)                                       # not before: a call that was refused has not written the token
        return out.view(B, 1, Hq, 128)[..., :D]

    def get_seq_length(self, layer_idx: Optional[int] = 0) -> int:
        self._config()
        L = self._layers[0 if layer_idx is None else layer_idx]
        return L.n_comp + L.n_res

    def get_mask_sizes(self, query_length: int, layer_idx: int = 0) -> Tuple[int, int]:
        """(kv_length, kv_offset) of the mask transformers builds before this layer's update."""
        return self.get_seq_length(layer_idx) + int(query_length), 0

    def compressed_bytes(self) -> int:
        """Bytes of packed streams held by all layers (synchronises, and checks the device status word)."""
        self.check_flags()
        n = 0
        for L in self._layers:
            if L.comp is not None:
                n += int(L.comp.k_bytes.sum().item()) + int(L.comp.v_bytes.sum().item())
        return n


# the reference keeps the implementation behind a second class name (packkv_quant.py:30)
PackKVCachePytorchQuant = PackKVCache
