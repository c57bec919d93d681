"""GPU: the cache class and its append path against the reference's cache state machine restated
on CPU (oracle/quant.py CacheLayerOracle: RoPE -> cut whole blocks -> quantise -> dequantise ->
cat).  Dense views must be bit-identical; fused attention within 2e-3."""
import pytest
import torch

from oracle import quant as Q
from packkv_b200 import cache as C
from packkv_b200 import ops, synth
from packkv_b200.config import PackKVCacheConfig, QuantMethod, RepackMethod

pytestmark = pytest.mark.gpu


def _cfg(method, k_rel=1 / 14, v_rel=1 / 14, hp=False, enable=True, repack=RepackMethod.NONE):
    return PackKVCacheConfig("synthetic", method, repack, hp, 64, 192, 16, k_rel, v_rel, enable_quant=enable)


def _modes(method):
    return {QuantMethod.KIVI: ("channel", "token"), QuantMethod.PackKV: ("token", "token")}[method]


@pytest.mark.parametrize("method,repack", [(QuantMethod.KIVI, RepackMethod.NONE), (QuantMethod.PackKV, RepackMethod.NONE),
                                           (QuantMethod.KIVI, RepackMethod.MEDIAN), (QuantMethod.PackKV, RepackMethod.MEDIAN)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_prefill_then_decode_matches_reference_cache(cuda_device, method, repack, dtype):
    dev = cuda_device
    B, H, G, S0, steps = 2, 2, 4, 333, 140
    cfg = _cfg(method, repack=repack)
    C.PackKVCacheConfigStatic.config = cfg
    try:
        cache = C.PackKVCache(B, H * G, 128, 1, materialize=True)
        km, vm = _modes(method)
        oracle = Q.CacheLayerOracle(64, 192, cfg.k_quant_scale_rel, cfg.v_quant_scale_rel, km, vm)
        k, v = synth.synth_kv(B, H, S0 + steps, 128, seed=31, dtype=dtype)
        cos, sin = synth.rope_tables(S0 + steps, 128, dtype=dtype)
        # prefill
        Ko, Vo = oracle.update(k[:, :, :S0], v[:, :, :S0], cos[:, :S0], sin[:, :S0])
        Kg, Vg = cache.update(k[:, :, :S0].to(dev), v[:, :, :S0].to(dev), 0, {"cos": cos[:, :S0].to(dev), "sin": sin[:, :S0].to(dev)})
        assert torch.equal(Kg.cpu(), Ko) and torch.equal(Vg.cpu(), Vo)
        assert cache.get_seq_length(0) == oracle.seq_length() == S0
        # decode: one token at a time; the residual stays within [128, 191]
        for t in range(S0, S0 + steps):
            Ko, Vo = oracle.update(k[:, :, t:t + 1], v[:, :, t:t + 1], cos[:, t:t + 1], sin[:, t:t + 1])
            Kg, Vg = cache.update(k[:, :, t:t + 1].to(dev), v[:, :, t:t + 1].to(dev), 0,
                                  {"cos": cos[:, t:t + 1].to(dev), "sin": sin[:, t:t + 1].to(dev)})
            assert 128 <= cache._layers[0].n_res <= 191
            assert cache.get_seq_length(0) == t + 1
            if (t - S0) % 16 == 0 or t == S0 + steps - 1:
                assert torch.equal(Kg.cpu(), Ko), t
                assert torch.equal(Vg.cpu(), Vo), t
                q = synth.synth_q(B, H * G, 128, seed=t, dtype=dtype)
                ref = Q.eager_attention(q, Ko, Vo).float()
                out = cache.attend(q.to(dev), 0).float().cpu()
                assert ((out - ref).abs().max() / ref.abs().max()).item() <= 2e-3, t
        cache.check_flags()
        assert cache.compressed_bytes() > 0
    finally:
        C.PackKVCacheConfigStatic.config = None


@pytest.mark.parametrize("method", [QuantMethod.KIVI, QuantMethod.PackKV])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_high_precision_zero_and_three_bit_cache(cuda_device, method, dtype):
    """high_precision_zero_point=True (zero = block minimum, utils/compute.py:97-101) with 3-bit scales:
    dense views bit-identical to the reference cache, fused attention within 2e-3."""
    dev = cuda_device
    B, H, G, S0, steps = 1, 2, 4, 260, 70
    cfg = _cfg(method, k_rel=1 / 6, v_rel=1 / 6, hp=True)
    C.PackKVCacheConfigStatic.config = cfg
    try:
        cache = C.PackKVCache(B, H * G, 128, 1, materialize=True)
        km, vm = _modes(method)
        oracle = Q.CacheLayerOracle(64, 192, 1 / 6, 1 / 6, km, vm, high_precision_zero=True)
        k, v = synth.synth_kv(B, H, S0 + steps, 128, seed=37, dtype=dtype)
        cos, sin = synth.rope_tables(S0 + steps, 128, dtype=dtype)
        Ko, Vo = oracle.update(k[:, :, :S0], v[:, :, :S0], cos[:, :S0], sin[:, :S0])
        Kg, Vg = cache.update(k[:, :, :S0].to(dev), v[:, :, :S0].to(dev), 0, {"cos": cos[:, :S0].to(dev), "sin": sin[:, :S0].to(dev)})
        assert torch.equal(Kg.cpu(), Ko) and torch.equal(Vg.cpu(), Vo)
        for t in range(S0, S0 + steps):
            Ko, Vo = oracle.update(k[:, :, t:t + 1], v[:, :, t:t + 1], cos[:, t:t + 1], sin[:, t:t + 1])
            Kg, Vg = cache.update(k[:, :, t:t + 1].to(dev), v[:, :, t:t + 1].to(dev), 0,
                                  {"cos": cos[:, t:t + 1].to(dev), "sin": sin[:, t:t + 1].to(dev)})
        assert torch.equal(Kg.cpu(), Ko) and torch.equal(Vg.cpu(), Vo)
        q = synth.synth_q(B, H * G, 128, seed=3, dtype=dtype)
        ref = Q.eager_attention(q, Ko, Vo).float()
        out = cache.attend(q.to(dev), 0).float().cpu()
        assert ((out - ref).abs().max() / ref.abs().max()).item() <= 2e-3
        cache.check_flags()
    finally:
        C.PackKVCacheConfigStatic.config = None


@pytest.mark.parametrize("method", [QuantMethod.KIVI, QuantMethod.PackKV])
@pytest.mark.parametrize("head_dim", [96, 64])
def test_head_dim_below_128_matches_reference_cache(cuda_device, method, head_dim):
    """Phi-3-style heads (head_dim 96, MHA): the cache stores them in 128-channel blocks whose tail repeats the
    first channels, which leaves every real channel's codes and parameters those of the reference's cache run on
    head_dim-wide tensors (models/phi.py:744-747 creates the cache with hidden_size // num_attention_heads).
    Dense views bit-identical, fused attention within 2e-3, prefill + decode across a block boundary."""
    dev, dtype = cuda_device, torch.bfloat16
    B, H, G, S0, steps, D = 2, 4, 1, 270, 70, head_dim
    cfg = _cfg(method)
    C.PackKVCacheConfigStatic.config = cfg
    try:
        cache = C.PackKVCache(B, H * G, D, 1, materialize=True)
        km, vm = _modes(method)
        oracle = Q.CacheLayerOracle(64, 192, cfg.k_quant_scale_rel, cfg.v_quant_scale_rel, km, vm)
        k, v = synth.synth_kv(B, H, S0 + steps, D, seed=41, dtype=dtype)
        cos, sin = synth.rope_tables(S0 + steps, D, dtype=dtype)
        Ko, Vo = oracle.update(k[:, :, :S0], v[:, :, :S0], cos[:, :S0], sin[:, :S0])
        Kg, Vg = cache.update(k[:, :, :S0].to(dev), v[:, :, :S0].to(dev), 0, {"cos": cos[:, :S0].to(dev), "sin": sin[:, :S0].to(dev)})
        assert Kg.shape[-1] == D and torch.equal(Kg.cpu(), Ko) and torch.equal(Vg.cpu(), Vo)
        for t in range(S0, S0 + steps):
            Ko, Vo = oracle.update(k[:, :, t:t + 1], v[:, :, t:t + 1], cos[:, t:t + 1], sin[:, t:t + 1])
            Kg, Vg = cache.update(k[:, :, t:t + 1].to(dev), v[:, :, t:t + 1].to(dev), 0,
                                  {"cos": cos[:, t:t + 1].to(dev), "sin": sin[:, t:t + 1].to(dev)})
        assert torch.equal(Kg.cpu(), Ko) and torch.equal(Vg.cpu(), Vo)
        q = synth.synth_q(B, H * G, D, seed=5, dtype=dtype)
        ref = Q.eager_attention(q, Ko, Vo).float()                  # scaling head_dim ** -0.5
        out = cache.attend(q.to(dev), 0).float().cpu()
        assert out.shape == ref.shape
        assert ((out - ref).abs().max() / ref.abs().max()).item() <= 2e-3
        cache.check_flags()
    finally:
        C.PackKVCacheConfigStatic.config = None


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_decode_step_append_inside_the_attention_launch(cuda_device, dtype):
    """A decode step without materialised K/V: update() only records the new token, attend() lets the attention
    launch rotate K, write both rows into the residual and attend over them.  The residual rows must equal the
    ones pkv_append_residual writes (bit for bit, same RoPE arithmetic), the attention output the reference's
    within 2e-3, and an update() that is not followed by attend() must still land in the residual."""
    dev = cuda_device
    B, H, G, S0, steps = 2, 2, 4, 300, 40
    cfg = _cfg(QuantMethod.KIVI)
    C.PackKVCacheConfigStatic.config = cfg
    try:
        fused, plain = C.PackKVCache(B, H * G, 128, 1), C.PackKVCache(B, H * G, 128, 1, materialize=True)
        oracle = Q.CacheLayerOracle(64, 192, cfg.k_quant_scale_rel, cfg.v_quant_scale_rel, "channel", "token")
        k, v = synth.synth_kv(B, H, S0 + steps, 128, seed=51, dtype=dtype)
        cos, sin = synth.rope_tables(S0 + steps, 128, dtype=dtype)
        kw = lambda a, b: {"cos": cos[:, a:b].to(dev), "sin": sin[:, a:b].to(dev)}
        Ko, Vo = oracle.update(k[:, :, :S0], v[:, :, :S0], cos[:, :S0], sin[:, :S0])
        for c in (fused, plain):
            c.update(k[:, :, :S0].to(dev), v[:, :, :S0].to(dev), 0, kw(0, S0))
        for t in range(S0, S0 + steps):
            Ko, Vo = oracle.update(k[:, :, t:t + 1], v[:, :, t:t + 1], cos[:, t:t + 1], sin[:, t:t + 1])
            n_comp_before = fused._layers[0].n_comp
            for c in (fused, plain):
                c.update(k[:, :, t:t + 1].to(dev), v[:, :, t:t + 1].to(dev), 0, kw(t, t + 1))
            if t % 3 == 0:
                continue                                             # no attend(): the next update() must flush the token
            # a step that moved a block out of the residual went through the ordinary path; every other step defers
            assert (fused._layers[0].pending is not None) == (fused._layers[0].n_comp == n_comp_before)
            q = synth.synth_q(B, H * G, 128, seed=t, dtype=dtype)
            out = fused.attend(q.to(dev), 0).float().cpu()
            assert fused._layers[0].pending is None
            ref = Q.eager_attention(q, Ko, Vo).float()
            assert ((out - ref).abs().max() / ref.abs().max()).item() <= 2e-3, t
            Lf, Lp = fused._layers[0], plain._layers[0]
            assert Lf.n_res == Lp.n_res
            assert torch.equal(Lf.k_res[:, :, : Lf.n_res], Lp.k_res[:, :, : Lp.n_res]), t
            assert torch.equal(Lf.v_res[:, :, : Lf.n_res], Lp.v_res[:, :, : Lp.n_res]), t
        Kd, Vd = fused.dense(0)
        assert torch.equal(Kd.cpu(), Ko) and torch.equal(Vd.cpu(), Vo)
        fused.check_flags()
    finally:
        C.PackKVCacheConfigStatic.config = None


def test_append_streams_equal_one_shot_encode(cuda_device):
    """Blocks appended one at a time give the same bytes as encoding the history in one call."""
    from packkv_b200 import encode, ops
    from packkv_b200.config import QuantMode
    dev = cuda_device
    C.PackKVCacheConfigStatic.config = _cfg(QuantMethod.KIVI)
    try:
        B, H, S = 2, 2, 64 * 9
        cache = C.PackKVCache(B, H, 128, 1)
        k, v = synth.synth_kv(B, H, S, 128, seed=5, dtype=torch.float16)
        cos, sin = synth.rope_tables(S, 128, dtype=torch.float16)
        cos1, sin1 = torch.ones_like(cos), torch.zeros_like(sin)      # identity rotation keeps K as is
        cache.update(k[:, :, :200].to(dev), v[:, :, :200].to(dev), 0, {"cos": cos1[:, :200].to(dev), "sin": sin1[:, :200].to(dev)})
        for t in range(200, S):
            cache.update(k[:, :, t:t + 1].to(dev), v[:, :, t:t + 1].to(dev), 0, {"cos": cos1[:, t:t + 1].to(dev), "sin": sin1[:, t:t + 1].to(dev)})
        L = cache._layers[0]
        n = L.n_comp
        assert n == S - 128 - S % 64 and n > 0
        one = encode.compress_kv(k[:, :, :n].to(dev), v[:, :, :n].to(dev), block=64, bits_k=4, bits_v=4, k_rel=1 / 14, v_rel=1 / 14,
                                 k_mode=QuantMode.ChannelQuant)
        torch.cuda.synchronize()
        for b in range(B):
            nk, nv = int(one.k_bytes[b].item()), int(one.v_bytes[b].item())
            assert int(L.comp.k_bytes[b].item()) == nk and int(L.comp.v_bytes[b].item()) == nv
            assert torch.equal(L.comp.k_stream[b, :nk], one.k_stream[b, :nk])
            assert torch.equal(L.comp.v_stream[b, :nv], one.v_stream[b, :nv])
        nkb, nvb = one.k_info.shape[1], one.v_info.shape[1]
        assert torch.equal(L.comp.k_info[:, : (n // 64) * H], one.k_info[:, : (n // 64) * H])
        assert torch.equal(L.comp.v_info[:, : (n // 64) * 2 * H], one.v_info[:, : (n // 64) * 2 * H])
    finally:
        C.PackKVCacheConfigStatic.config = None


def test_config_contract_and_disabled_quant(cuda_device):
    dev = cuda_device
    C.PackKVCacheConfigStatic.config = None
    cache = C.PackKVCache(1, 8, 128, 2)
    k, v = synth.synth_kv(1, 2, 10, 128, seed=1, dtype=torch.float16)
    cos, sin = synth.rope_tables(10, 128, dtype=torch.float16)
    kw = {"cos": cos.to(dev), "sin": sin.to(dev)}
    with pytest.raises(ValueError):                     # packkv_quant.py:54-55
        cache.update(k.to(dev), v.to(dev), 0, kw)
    with pytest.raises(ValueError):
        cache.get_seq_length(0)
    C.PackKVCacheConfigStatic.config = _cfg(QuantMethod.KIVI, enable=False)
    try:
        K, V = cache.update(k.to(dev), v.to(dev), 1, kw)
        assert torch.equal(K.cpu(), Q.rope(k, cos, sin)) and torch.equal(V.cpu(), v)
        K, V = cache.update(k[:, :, :1].to(dev), v[:, :, :1].to(dev), 1, {"cos": cos[:, :1].to(dev), "sin": sin[:, :1].to(dev)})
        assert K.shape[2] == 11 and cache.get_seq_length(1) == 11 and cache.get_seq_length(0) == 0
    finally:
        C.PackKVCacheConfigStatic.config = None
    cfg = _cfg(QuantMethod.KIVI, k_rel=0.1, v_rel=0.2)
    assert PackKVCacheConfig.from_str(str(cfg)) == cfg and hash(PackKVCacheConfig.from_str(str(cfg))) == hash(cfg)
    assert C.bits_for_rel(0.1) == 4 and C.bits_for_rel(0.2) == 3 and C.bits_for_rel(1 / 14) == 4 and C.bits_for_rel(0.5) == 2


@pytest.mark.parametrize("D", [128, 96])
@pytest.mark.parametrize("repack", [RepackMethod.NONE, RepackMethod.MEDIAN])
def test_prompts_in_pieces_match_reference_cache(cuda_device, D, repack):
    """Pieces that leave the residual short of a block, fill it past its capacity (300 tokens behind 130 of 256 rows), cross
    a block boundary one token at a time, and end on it, from strided projections: dense rows bit-identical."""
    dev, dtype, B, H = cuda_device, torch.bfloat16, 2, 2
    cfg = _cfg(QuantMethod.KIVI, repack=repack)
    C.PackKVCacheConfigStatic.config = cfg
    try:
        cache = C.PackKVCache(B, H, D, 1, materialize=True)
        oracle = Q.CacheLayerOracle(64, 192, cfg.k_quant_scale_rel, cfg.v_quant_scale_rel, "channel", "token")
        pieces = [30, 100, 300, 1, 40, 1, 64]
        k, v = synth.synth_kv(B, H, sum(pieces), D, seed=12, dtype=dtype)
        cos, sin = synth.rope_tables(sum(pieces), D, dtype=dtype)
        t = 0
        for n in pieces:
            def part(x):
                return x[:, :, t:t + n]
            Ko, Vo = oracle.update(part(k), part(v), cos[:, t:t + n], sin[:, t:t + n])
            Kg, Vg = cache.update(*(part(x).to(dev).transpose(1, 2).contiguous().transpose(1, 2) for x in (k, v)), 0,
                                  {"cos": cos[:, t:t + n].to(dev), "sin": sin[:, t:t + n].to(dev)})
            assert torch.equal(Kg.cpu(), Ko) and torch.equal(Vg.cpu(), Vo), t
            t += n
        cache.check_flags()
    finally:
        C.PackKVCacheConfigStatic.config = None


@pytest.mark.parametrize("D", [128, 96])
def test_update_refuses_rotation_tables_of_another_length(cuda_device, D):
    dev, dtype = cuda_device, torch.bfloat16
    C.PackKVCacheConfigStatic.config = _cfg(QuantMethod.KIVI)
    try:
        cache = C.PackKVCache(1, 2, D, 1)
        cos, sin = synth.rope_tables(500, D, device=dev, dtype=dtype)
        for T in (400, 10, 1):                               # a prompt that is packed, tokens that stay behind, a decode step
            k, v = synth.synth_kv(1, 2, T, D, seed=5, dtype=dtype, device=dev)
            for n in (T + 1, 500):
                with pytest.raises(ValueError):
                    cache.update(k, v, 0, {"cos": cos[:, :n], "sin": sin[:, :n]})
                    cache.flush()
            if T > 1:
                cache.update(k, v, 0, {"cos": cos[:, :T], "sin": sin[:, :T]})
    finally:
        C.PackKVCacheConfigStatic.config = None


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 72, 96, 120])
@pytest.mark.parametrize("tables", ["row", "rows", None])
def test_narrow_decode_step_inside_the_attention_launch(cuda_device, D, dtype, tables):
    """Heads below 128 channels: an attention launch that is handed the step's token widens its rows and reads the narrow q.  Residual rows bit
    for bit those of widen_rows (halves of 32 .. 60 channels, rows at odd addresses, tables for one or all sequences), outputs those of a q that
    is padded and rows that are written beforehand, with and without packed blocks.  A cache writes the rows in update(), with and without an
    attend() between two steps."""
    dev, B, H, G = cuda_device, 2, 2, 3
    C.PackKVCacheConfigStatic.config = _cfg(QuantMethod.PackKV)
    try:
        for S0 in (3, 270):
            cache = C.PackKVCache(B, H * G, D, 1)
            cache._scratch = ops.new_attention_scratch(dev)
            k, v = synth.synth_kv(B, H, S0, D, seed=S0, dtype=dtype, device=dev)
            cache.update(k, v, 0)
            for t in range(5):
                gen = torch.Generator(device=dev).manual_seed(t)
                buf = torch.randn(2, B, H, D + 1, generator=gen, device=dev).to(dtype)
                kn, vn = (x[..., t % 2: t % 2 + D].unsqueeze(2) for x in buf)
                q = torch.randn(B, H * G, 1, D, generator=gen, device=dev).to(dtype)
                kw = None
                if tables:
                    cs = torch.randn(2, B if tables == "rows" else 1, 1, D, generator=gen, device=dev).to(dtype)
                    kw = {"cos": cs[0], "sin": cs[1]}
                cache.update(kn, vn, 0, kw)
                assert cache._layers[0].pending is None
                if t == 2:
                    continue
                wide = torch.zeros(B, H * G, 128, dtype=dtype, device=dev)
                wide[..., :D] = q[:, :, 0]
                L = cache._layers[0]
                layer = L.comp if L.n_comp else None
                want = ops.decode_attention(wide, layer, L.k_res, L.v_res, L.n_res, scaling=D ** -0.5, kv_heads=H, scratch=cache._scratch)
                got = cache.attend(q, 0)
                assert got.shape == (B, 1, H * G, D) and torch.equal(got[:, 0], want[..., :D])
                k_res, v_res = L.k_res.clone(), L.v_res.clone()
                k_res[:, :, L.n_res - 1], v_res[:, :, L.n_res - 1] = float("nan"), float("nan")
                got = ops.decode_attention_narrow(q[:, :, 0].contiguous(), layer, k_res, v_res, L.n_res, scaling=D ** -0.5, kv_heads=H, scratch=cache._scratch,
                                                  append=(kn, vn, *(cs if tables else (None, None))))
                assert torch.equal(got[..., :D], want[..., :D])
                assert torch.equal(k_res[:, :, : L.n_res], L.k_res[:, :, : L.n_res]) and torch.equal(v_res[:, :, : L.n_res], L.v_res[:, :, : L.n_res])
            cache.check_flags()
        other = torch.randn(B, H * G, 1, 128, device=dev).to(dtype)
        L = cache._layers[0]
        want = ops.decode_attention(other[:, :, 0], L.comp, L.k_res, L.v_res, L.n_res, kv_heads=H, scratch=cache._scratch)
        assert torch.equal(cache.attend(other, 0)[:, 0], want)           # a wider query than the rows of the step
    finally:
        C.PackKVCacheConfigStatic.config = None


def test_steps_from_one_buffer(cuda_device):
    """A caller that keeps one projection buffer and one pair of table rows for all steps of 128 channels, and writes them again once attend(),
    flush() or dense() has been called for the step before."""
    dev, dtype, B, H, G, steps = cuda_device, torch.bfloat16, 2, 2, 4, 6
    C.PackKVCacheConfigStatic.config = _cfg(QuantMethod.KIVI)
    try:
        one, own = C.PackKVCache(B, H * G, 128, 1), C.PackKVCache(B, H * G, 128, 1)
        k, v = synth.synth_kv(B, H, 300 + steps, 128, seed=3, dtype=dtype, device=dev)
        cos, sin = synth.rope_tables(300 + steps, 128, device=dev, dtype=dtype)
        for cache in (one, own):
            cache.update(k[:, :, :300], v[:, :, :300], 0, {"cos": cos[:, :300], "sin": sin[:, :300]})
        buf = [torch.empty(B, H, 1, 128, dtype=dtype, device=dev) for _ in range(2)] + [torch.empty(1, 1, 128, dtype=dtype, device=dev) for _ in range(2)]
        for n in range(steps):
            t = 300 + n
            row = [k[:, :, t:t + 1].clone(), v[:, :, t:t + 1].clone(), cos[:, t:t + 1].clone(), sin[:, t:t + 1].clone()]
            for b, x in zip(buf, row):
                b.copy_(x)
            one.update(buf[0], buf[1], 0, {"cos": buf[2], "sin": buf[3]})
            own.update(row[0], row[1], 0, {"cos": row[2], "sin": row[3]})
            q = synth.synth_q(B, H * G, 128, seed=n, dtype=dtype).to(dev)
            if n % 3 == 0:
                assert torch.equal(one.attend(q, 0), own.attend(q, 0)), n
            elif n % 3 == 1:
                one.flush()
            else:
                one.dense(0)
            for b in buf:
                b.fill_(float("nan"))
        own.flush()
        a, b = one._layers[0], own._layers[0]
        assert a.n_res == b.n_res and torch.equal(a.k_res[:, :, : a.n_res], b.k_res[:, :, : b.n_res]) and torch.equal(a.v_res[:, :, : a.n_res], b.v_res[:, :, : b.n_res])
    finally:
        C.PackKVCacheConfigStatic.config = None


@pytest.mark.parametrize("D", [64, 96])
def test_narrow_steps_from_one_buffer(cuda_device, D):
    """A caller that keeps one projection buffer and one pair of table rows for all steps of a narrow-headed model: update() has taken what they
    held when it was called, whether attend() follows, follows after the buffers are written again, or not at all."""
    dev, dtype, B, H, G, steps = cuda_device, torch.bfloat16, 2, 2, 4, 6
    C.PackKVCacheConfigStatic.config = _cfg(QuantMethod.KIVI)
    try:
        one, own = C.PackKVCache(B, H * G, D, 1), C.PackKVCache(B, H * G, D, 1)
        k, v = synth.synth_kv(B, H, 300 + steps, D, seed=3, dtype=dtype, device=dev)
        cos, sin = synth.rope_tables(300 + steps, D, device=dev, dtype=dtype)
        for cache in (one, own):
            cache.update(k[:, :, :300], v[:, :, :300], 0, {"cos": cos[:, :300], "sin": sin[:, :300]})
        buf = [torch.empty(B, H, 1, D, dtype=dtype, device=dev) for _ in range(2)] + [torch.empty(1, 1, D, dtype=dtype, device=dev) for _ in range(2)]
        for n in range(steps):
            t = 300 + n
            row = [k[:, :, t:t + 1].clone(), v[:, :, t:t + 1].clone(), cos[:, t:t + 1].clone(), sin[:, t:t + 1].clone()]
            for b, x in zip(buf, row):
                b.copy_(x)
            one.update(buf[0], buf[1], 0, {"cos": buf[2], "sin": buf[3]})
            own.update(row[0], row[1], 0, {"cos": row[2], "sin": row[3]})
            if n % 3 != 2:
                if n % 3 == 1:
                    for b in buf:
                        b.fill_(float("nan"))
                q = synth.synth_q(B, H * G, D, seed=n, dtype=dtype).to(dev)
                assert torch.equal(one.attend(q, 0), own.attend(q, 0)), n
        a, b = one._layers[0], own._layers[0]
        assert a.n_res == b.n_res and torch.equal(a.k_res[:, :, : a.n_res], b.k_res[:, :, : b.n_res]) and torch.equal(a.v_res[:, :, : a.n_res], b.v_res[:, :, : b.n_res])
    finally:
        C.PackKVCacheConfigStatic.config = None


@pytest.mark.parametrize("D", [96, 128])
def test_refused_attend_keeps_the_step(cuda_device, D):
    """An attend() that is refused (a query of another type, q heads that are no multiple of the KV heads, a group above 8) leaves the step's
    token in place: the attend() that is corrected, dense() and the next steps find its row."""
    dev, dtype, B, H = cuda_device, torch.float16, 2, 2
    C.PackKVCacheConfigStatic.config = _cfg(QuantMethod.KIVI)
    try:
        cache, plain = C.PackKVCache(B, H * 2, D, 1), C.PackKVCache(B, H * 2, D, 1)
        k, v = synth.synth_kv(B, H, 303, D, seed=4, dtype=dtype, device=dev)
        cos, sin = synth.rope_tables(303, D, device=dev, dtype=dtype)
        kw = lambda a, b: {"cos": cos[:, a:b], "sin": sin[:, a:b]}
        for c in (cache, plain):
            c.update(k[:, :, :300], v[:, :, :300], 0, kw(0, 300))
        for t in range(300, 303):
            q = synth.synth_q(B, H * 2, D, seed=t, dtype=dtype).to(dev)
            for c in (cache, plain):
                c.update(k[:, :, t:t + 1], v[:, :, t:t + 1], 0, kw(t, t + 1))
            plain.flush()
            L = cache._layers[0]
            if L.pending is not None:                    # what the row holds until the launch writes it
                L.k_res[:, :, L.n_res - 1], L.v_res[:, :, L.n_res - 1] = 7.0, 7.0
            for bad in (q.bfloat16(), q[:, :3], q.repeat(1, 5, 1, 1)[:, : H * 9]):
                with pytest.raises((ValueError, RuntimeError)):
                    cache.attend(bad, 0)
            if t == 301:
                assert all(torch.equal(a, b) for a, b in zip(cache.dense(0), plain.dense(0)))
            else:
                assert torch.equal(cache.attend(q, 0), plain.attend(q, 0))
        a, b = cache._layers[0], plain._layers[0]
        assert torch.equal(a.k_res[:, :, : a.n_res], b.k_res[:, :, : b.n_res]) and torch.equal(a.v_res[:, :, : a.n_res], b.v_res[:, :, : b.n_res])
    finally:
        C.PackKVCacheConfigStatic.config = None


@pytest.mark.parametrize("form", ["odd address", "odd strides", "v channels apart", "v of another type", "tables of another type", "tables apart", "k of another type", "heads"])
def test_step_that_the_attention_launch_does_not_take(cuda_device, form):
    """A step of 128 channels whose tensors the attention launch cannot read as they are: written (converted) by update() like a step of any
    other length, or refused there, with the token not counted and the cache as it was."""
    dev, dtype, B, H, G = cuda_device, torch.bfloat16, 2, 2, 2
    C.PackKVCacheConfigStatic.config = _cfg(QuantMethod.KIVI)
    try:
        cache, plain = C.PackKVCache(B, H * G, 128, 1), C.PackKVCache(B, H * G, 128, 1)
        k, v = synth.synth_kv(B, H, 301, 128, seed=6, dtype=dtype, device=dev)
        cos, sin = synth.rope_tables(301, 128, device=dev, dtype=dtype)
        for c in (cache, plain):
            c.update(k[:, :, :300], v[:, :, :300], 0, {"cos": cos[:, :300], "sin": sin[:, :300]})
        row = [k[:, :, 300:].clone(), v[:, :, 300:].clone(), cos[:, 300:].clone(), sin[:, 300:].clone()]
        plain.update(row[0], row[1], 0, {"cos": row[2], "sin": row[3]})
        plain.flush()
        if form == "odd address":
            row[0] = torch.empty(B * H * 128 + 1, dtype=dtype, device=dev)[1:].view(B, H, 1, 128).copy_(row[0])
        elif form == "odd strides":
            row[1] = torch.empty(B, H, 1, 129, dtype=dtype, device=dev)[..., :128].copy_(row[1])
        elif form == "v channels apart":
            row[1] = torch.empty(B, H, 1, 128, 2, dtype=dtype, device=dev)[..., 0].copy_(row[1])
        elif form == "v of another type":
            row[1] = row[1].float()
        elif form == "tables of another type":
            row[2], row[3] = row[2].float(), row[3].float()
        elif form == "tables apart":
            row[2] = torch.empty(1, 1, 128, 2, dtype=dtype, device=dev)[..., 0].copy_(row[2])
        q = synth.synth_q(B, H * G, 128, seed=1, dtype=dtype).to(dev)
        if form in ("k of another type", "heads"):
            bad = row[0].half() if form[0] == "k" else row[0].repeat(1, 2, 1, 1)
            with pytest.raises(ValueError):
                cache.update(bad, row[1].half() if form[0] == "k" else row[1].repeat(1, 2, 1, 1), 0, {"cos": row[2], "sin": row[3]})
            assert cache.get_seq_length(0) == 300 and cache._layers[0].pending is None
            cache.update(row[0], row[1], 0, {"cos": row[2], "sin": row[3]})
        else:
            cache.update(row[0], row[1], 0, {"cos": row[2], "sin": row[3]})
            assert cache._layers[0].pending is None
        assert torch.equal(cache.attend(q, 0), plain.attend(q, 0))
        a, b = cache._layers[0], plain._layers[0]
        assert a.n_res == b.n_res and torch.equal(a.k_res[:, :, : a.n_res], b.k_res[:, :, : b.n_res]) and torch.equal(a.v_res[:, :, : a.n_res], b.v_res[:, :, : b.n_res])
    finally:
        C.PackKVCacheConfigStatic.config = None


@pytest.mark.parametrize("flush", [False, True])
def test_update_and_attend_on_two_streams(cuda_device, flush):
    """A step goes to update() on one stream, to attend() (or flush()) on another that is ordered behind it and busy, and its tensors are let go:
    the first stream's next tensors must not get their memory before the row is written."""
    dev, dtype, B, H, G = cuda_device, torch.bfloat16, 2, 2, 2
    C.PackKVCacheConfigStatic.config = _cfg(QuantMethod.KIVI)
    try:
        cache, plain = C.PackKVCache(B, H * G, 128, 1), C.PackKVCache(B, H * G, 128, 1)
        k, v = synth.synth_kv(B, H, 301, 128, seed=6, dtype=dtype, device=dev)
        cos, sin = synth.rope_tables(301, 128, device=dev, dtype=dtype)
        for c in (cache, plain):
            c.update(k[:, :, :300], v[:, :, :300], 0, {"cos": cos[:, :300], "sin": sin[:, :300]})
        plain.update(k[:, :, 300:], v[:, :, 300:], 0, {"cos": cos[:, 300:], "sin": sin[:, 300:]})
        q = synth.synth_q(B, H * G, 128, seed=1, dtype=dtype).to(dev)
        want = plain.attend(q, 0)
        plain.flush()
        torch.cuda.synchronize()
        first, second = torch.cuda.Stream(), torch.cuda.Stream()
        with torch.cuda.stream(second):
            cache.attend(q, 0)                                     # buffers and kernels are there: nothing below waits for an allocation
        torch.full((1,), float("nan"), dtype=dtype, device=dev)
        torch.cuda.synchronize()
        with torch.cuda.stream(first):
            row = [k[:, :, 300:].clone(), v[:, :, 300:].clone(), cos[:, 300:].clone(), sin[:, 300:].clone()]
            cache.update(row[0], row[1], 0, {"cos": row[2], "sin": row[3]})
            shapes = [t.shape for t in row]
            del row
        assert cache._layers[0].pending is not None
        second.wait_stream(first)
        with torch.cuda.stream(second):
            torch.cuda._sleep(20_000_000)                          # about 10 ms
            got = cache.flush() if flush else cache.attend(q, 0)
        with torch.cuda.stream(first):
            new = [torch.full(s, float("nan"), dtype=dtype, device=dev) for s in shapes for _ in range(4)]
        torch.cuda.synchronize()
        del new
        a, b = cache._layers[0], plain._layers[0]
        assert torch.equal(a.k_res[:, :, : a.n_res], b.k_res[:, :, : b.n_res]) and torch.equal(a.v_res[:, :, : a.n_res], b.v_res[:, :, : b.n_res])
        assert flush or torch.equal(got, want)
    finally:
        C.PackKVCacheConfigStatic.config = None
