"""The work that programs have this library do, as measurable cases.

Four kinds of work, each through its public entry points:

decode    a serving engine's decode step over `layers` layers: ops.decode_attention on the packed streams with the step's
          new token folded in (append) and the engine's scratch, output and flag buffers.
session   a model's use of PackKVCache: a prompt goes through update() of every layer (which returns the dense K and V that
          the prompt's own attention needs), then `new_tokens` decode steps of update() + attend(), or, with
          materialize, of update() alone, which returns dense K and V as the reference's cache does.
encode    an engine packs K and V of prompts, or of the blocks that leave the residual, into stream buffers that it keeps
          (ops.encode_tensor; with median reorder ops.value_median_order before it).
harness   the packkv_cuda functions in the order in which the reference's evaluation calls them: codes on the host are
          encoded, decoded again, and the packed streams multiplied with a query (K) or with weights (V) on the GPU.

Values are packkv_b200.synth's: per-channel lognormal scales with a few outlier channels for K, normal V and queries.
"""
import math

import torch

import packkv_cuda
from packkv_b200 import cache, encode, ops, synth
from packkv_b200.config import PackKVCacheConfig, QuantMethod, QuantMode, RepackMethod

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
RECENT = 192             # residual buffer of the reference's scripts: 128..191 tokens stay uncompressed with 64-token blocks
U32 = getattr(torch, "uint32", torch.int32)


def _decode(layers, batch, kv_heads, group, ctx, dtype="bf16", bits_k=4, bits_v=4, block=64, v_block=128, k_quant="channel"):
    return dict(kind="decode", layers=layers, batch=batch, kv_heads=kv_heads, group=group, ctx=ctx, dtype=dtype, bits_k=bits_k, bits_v=bits_v,
                block=block, v_block=v_block, k_quant=k_quant)


def _session(layers, batch, kv_heads, group, head_dim, prompt, new_tokens, dtype="bf16", k_rel=0.1, v_rel=0.2, block=64, method="KIVI",
             repack="none", materialize=False):
    return dict(kind="session", layers=layers, batch=batch, kv_heads=kv_heads, group=group, head_dim=head_dim, prompt=prompt, new_tokens=new_tokens,
                dtype=dtype, k_rel=k_rel, v_rel=v_rel, block=block, method=method, repack=repack, materialize=materialize)


def _encode(layers, batch, kv_heads, tokens, dtype="fp16", bits_k=4, bits_v=4, block=64, v_block=64, k_quant="channel", repack="none", layout="bhsd"):
    return dict(kind="encode", layers=layers, batch=batch, kv_heads=kv_heads, tokens=tokens, dtype=dtype, bits_k=bits_k, bits_v=bits_v, block=block,
                v_block=v_block, k_quant=k_quant, repack=repack, layout=layout)


def _harness(ctx, hidden, dtype="fp16", bits_k=4, bits_v=3):
    return dict(kind="harness", ctx=ctx, hidden=hidden, dtype=dtype, bits_k=bits_k, bits_v=bits_v)


def listed():
    return [
        # one chat turn on a short context: nothing but launch latency and host work
        dict(_decode(4, 1, 8, 4, 700), name="decode 1 x 700"),
        # one long document (the reference's own throughput scripts run one sequence)
        dict(_decode(2, 1, 8, 4, 32768), name="decode 1 x 32k"),
        # the ordinary serving batch: Llama-3.1-8B-shaped, 16 sequences of 8192 tokens
        dict(_decode(2, 16, 8, 4, 8192), name="decode 16 x 8k"),
        # the long-context serving batch: Qwen3-8B-shaped, 2-bit K, 128-token blocks
        dict(_decode(1, 8, 8, 4, 32768, bits_k=2, block=128), name="decode 8 x 32k 2-bit"),
        # one rank of a head-sharded model, odd sizes: two KV heads of seven q heads each, K parameters per token, 3 bits, 64-token V blocks
        dict(_decode(3, 5, 2, 7, 5333, dtype="fp16", bits_k=3, bits_v=3, v_block=64, k_quant="token"), name="decode 5 x 5333 token"),
        # a short conversation: prompt and answer of two sequences through the cache class, four layers
        dict(_session(4, 2, 8, 4, 128, 777, 96), name="session 777 + 96"),
        # a long prompt and its first token (time to first token)
        dict(_session(2, 4, 8, 4, 128, 8191, 1), name="session 8191 + 1"),
        # Phi-3-mini-shaped: 32 KV heads of 96 channels without grouping, per-token K, across a block boundary
        dict(_session(2, 4, 32, 1, 96, 1025, 70, method="PackKV"), name="session 96-wide heads"),
        # the blocks of 64 tokens that leave the residual of 16 sequences in one decode step, four layers
        dict(_encode(4, 16, 8, 64), name="encode one block"),
        # prompts of a serving batch packed with the median reorder
        dict(_encode(1, 4, 8, 8192, dtype="bf16", repack="median"), name="encode 4 x 8k median"),
        # Mistral-7B-shaped prefill encode
        dict(_encode(1, 8, 8, 16384), name="encode 8 x 16k"),
        # the reference's evaluation loop for one layer's K and V, codes on the host
        dict(_harness(8192, 1024), name="harness 8192 x 1024"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "session", "session", "encode", "encode", "harness"])
    dtype = rng.choice(["bf16", "fp16"])
    k_quant = rng.choice(["channel", "channel", "token"])
    heads = rng.choice([1, 2, 4, 8, 8, 8])
    if kind == "decode":
        block = rng.choice([64, 64, 64, 128])
        v_block = 128 if block == 128 else rng.choice([64, 128])
        ctx = _log(rng, 400, 32768)
        layers, group = rng.randint(1, 4), rng.choice([1, 2, 4, 4, 6, 7, 8])
        most = max(1, min(48, 8 * 8 * 32768 // (layers * heads * ctx)))
        return _decode(layers, _log(rng, 1, most), heads, group, ctx, dtype, rng.choice([2, 3, 4, 4]), rng.choice([2, 3, 4, 4]), block, v_block, k_quant)
    if kind == "session":
        layers, head_dim = rng.randint(1, 4), rng.choice([128, 128, 128, 96, 64])
        prompt = _log(rng, 100, 8191)
        most = max(1, min(16, 4 * 8 * 8191 * 2 // (layers * heads * prompt)))
        batch = _log(rng, 1, most)
        materialize = rng.random() < 0.2
        step = layers * batch * heads * prompt           # rows that a decode step reads; a dense step also writes them
        new = min(rng.randint(1, 60 // (2 * layers) - 1), max(1, 3_000_000 // step)) if materialize else min(_log(rng, 1, 384 // layers), max(1, 16_000_000 // step))
        k_rel, v_rel = rng.choice([(0.1, 0.2), (0.1, 0.2), (1 / 14, 1 / 14), (0.5, 1 / 14)])
        return _session(layers, batch, heads, rng.choice([1, 2, 4, 4, 8]), head_dim, prompt, new, dtype, k_rel, v_rel, 64, rng.choice(["KIVI", "PackKV"]),
                        rng.choice(["none", "none", "none", "median"]), materialize)
    if kind == "encode":
        repack = rng.choice(["none", "none", "median"])
        block = 64 if repack == "median" else rng.choice([64, 64, 64, 128])
        v_block = rng.choice([block, block, 128])
        layers = rng.randint(1, 4)
        tokens = v_block * _log(rng, 1, 16384 // v_block)
        most = max(1, min(32, 8 * 8 * 16384 // (layers * heads * tokens)))
        return _encode(layers, _log(rng, 1, most), heads, tokens, dtype, rng.choice([2, 3, 4, 4]), rng.choice([2, 3, 4, 4]), block, v_block, k_quant,
                       repack, rng.choice(["bhsd", "bshd"]))
    return _harness(128 * _log(rng, 4, 64), 128 * rng.choice([1, 2, 4, 8]), dtype, rng.choice([3, 4]), rng.choice([3, 4]))


# ---- what a program has in hand before the call -------------------------------------------------------------------------
def _split(ctx, block):
    """Compressed and residual tokens of a context, by the cache's cut rule."""
    n = cache.compress_block_count(ctx, block, RECENT) * block
    return n, ctx - n


def _k_mode(case):
    return QuantMode.ChannelQuant if case["k_quant"] == "channel" else QuantMode.TokenQuant


def _rows(gen, *shape, dtype):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32).to(dtype)


def _prepare_decode(case, seed):
    dtype, B, H, G = DTYPES[case["dtype"]], case["batch"], case["kv_heads"], case["group"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n_comp, n_res = _split(case["ctx"], max(case["block"], case["v_block"]))
    layers = []
    for li in range(case["layers"]):
        k, v = synth.synth_kv(B, H, case["ctx"], 128, seed=seed * 64 + li, dtype=dtype, device="cuda", apply_rope=True)
        layer = None
        if n_comp:
            layer = encode.compress_kv(k[:, :, :n_comp], v[:, :, :n_comp], block=case["block"], bits_k=case["bits_k"], bits_v=case["bits_v"],
                                       k_rel=synth.rel_for_bits(case["bits_k"]), v_rel=synth.rel_for_bits(case["bits_v"]), k_mode=_k_mode(case),
                                       cbk=case["block"], cbv=case["v_block"])
            for name in ("k", "v"):                 # keep what is used of the streams, in 16-byte multiples
                used = (int(getattr(layer, name + "_bytes").max().item()) + 31) // 16 * 16
                setattr(layer, name + "_stream", getattr(layer, name + "_stream")[:, :used].contiguous())
        k_res = torch.zeros(B, H, RECENT + 128, 128, dtype=dtype, device="cuda")
        v_res = torch.zeros_like(k_res)
        k_res[:, :, : n_res - 1], v_res[:, :, : n_res - 1] = k[:, :, n_comp:-1], v[:, :, n_comp:-1]
        # the step's projections as a model hands them over: (B, 1, heads, 128) seen as (B, heads, 1, 128)
        k_new, v_new = (_rows(gen, B, 1, H, 128, dtype=dtype).transpose(1, 2) for _ in range(2))
        layers.append((layer, k_res, v_res, k_new, v_new, _rows(gen, B, H * G, 128, dtype=dtype)))
        del k, v
    cos, sin = synth.rope_tables(1, 128, start=case["ctx"] - 1, device="cuda", dtype=dtype)
    return dict(layers=layers, n_res=n_res, kv_heads=H, cos=cos, sin=sin, flags=ops.new_flags("cuda"), scratch=ops.new_attention_scratch("cuda"),
                outs=[torch.empty_like(layer[5]) for layer in layers])


def _run_decode(s):
    for (layer, k_res, v_res, k_new, v_new, q), out in zip(s["layers"], s["outs"]):
        ops.decode_attention(q, layer, k_res, v_res, s["n_res"], out=out, flags=s["flags"], kv_heads=s["kv_heads"],
                             append=(k_new, v_new, s["cos"], s["sin"]), scratch=s["scratch"])
    return {"out": s["outs"], "k_res": [x[1] for x in s["layers"]], "v_res": [x[2] for x in s["layers"]], "flags": s["flags"]}


def _prepare_session(case, seed):
    dtype, B, H, D = DTYPES[case["dtype"]], case["batch"], case["kv_heads"], case["head_dim"]
    S, N = case["prompt"], case["new_tokens"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    prompts, steps = [], []
    for li in range(case["layers"]):
        k, v = synth.synth_kv(B, H, S, D, seed=seed * 64 + li, dtype=dtype, device="cuda")
        # (B, S, heads, D) in memory, as the projections write it, seen as (B, heads, S, D)
        prompts.append(tuple(t.transpose(1, 2).contiguous().transpose(1, 2) for t in (k, v)))
        k, v = _rows(gen, N, B, 1, H, D, dtype=dtype), _rows(gen, N, B, 1, H, D, dtype=dtype)
        q = _rows(gen, N, B, 1, H * case["group"], D, dtype=dtype)
        steps.append([tuple(t[n].transpose(1, 2) for t in (k, v, q)) for n in range(N)])
    cos, sin = synth.rope_tables(S + N, D, device="cuda", dtype=dtype)
    rope = [{"cos": cos[:, t:t + n], "sin": sin[:, t:t + n]} for t, n in [(0, S)] + [(S + n, 1) for n in range(N)]]
    config = PackKVCacheConfig("synthetic", QuantMethod[case["method"]], RepackMethod[case["repack"].upper()], False, case["block"], RECENT, 16,
                               case["k_rel"], case["v_rel"])
    return dict(case=case, config=config, prompts=prompts, steps=steps, rope=rope)


def _run_session(s):
    case = s["case"]
    cache.PackKVCacheConfigStatic.config = s["config"]
    kv = cache.PackKVCache(case["batch"], case["kv_heads"] * case["group"], case["head_dim"], case["layers"], materialize=case["materialize"])
    dense = [kv.update(k, v, li, s["rope"][0]) for li, (k, v) in enumerate(s["prompts"])]
    outs = []
    for n in range(case["new_tokens"]):
        for li in range(case["layers"]):
            k, v, q = s["steps"][li][n]
            got = kv.update(k, v, li, s["rope"][1 + n])
            outs.append(got if case["materialize"] else kv.attend(q, li))
    return {"prompt": dense, "steps": outs if case["materialize"] else torch.stack(outs)}


def _prepare_encode(case, seed):
    dtype, B, H, S = DTYPES[case["dtype"]], case["batch"], case["kv_heads"], case["tokens"]
    layers = []
    for li in range(case["layers"]):
        kv = synth.synth_kv(B, H, S, 128, seed=seed * 64 + li, dtype=dtype, device="cuda", apply_rope=True)
        if case["layout"] == "bshd":
            kv = tuple(t.transpose(1, 2).contiguous().transpose(1, 2) for t in kv)
        stores = {}
        for which, bits, cb in (("k", case["bits_k"], case["block"]), ("v", case["bits_v"], case["v_block"])):
            channel = which == "k" and case["k_quant"] == "channel"
            shape = (B, H, S // case["block"], 128) if channel else (B, S)
            stores[which] = dict(scale=torch.zeros(shape, dtype=dtype, device="cuda"), zero=torch.zeros(shape, dtype=dtype, device="cuda"),
                                 stream=torch.zeros(B, encode.stream_capacity(which, S, H, cb, bits), dtype=torch.uint8, device="cuda"),
                                 info=torch.zeros(B, (S // cb) * H * (1 if which == "k" else 2), 2, dtype=torch.int32, device="cuda"),
                                 stream_bytes=torch.zeros(B, dtype=torch.int32, device="cuda"))
        layers.append((kv, stores))
    return dict(case=case, layers=layers, flags=ops.new_flags("cuda"), scratch=torch.zeros(B * S * H * 128, dtype=torch.uint8, device="cuda"),
                mode=ops.K_CHANNEL if case["k_quant"] == "channel" else ops.K_TOKEN)


def _run_encode(s):
    case, orders = s["case"], []
    for (k, v), stores in s["layers"]:
        more = dict(flags=s["flags"], scratch=s["scratch"])
        v_rel = synth.rel_for_bits(case["bits_v"])
        if case["repack"] == "median":
            orders.append(ops.value_median_order(v, case["block"], v_rel, flags=s["flags"]))
            more.update(order=orders[-1], order_block=case["block"])
        ops.encode_tensor("k", k, case["block"], synth.rel_for_bits(case["bits_k"]), s["mode"], case["bits_k"], case["block"], **stores["k"], **more)
        ops.encode_tensor("v", v, case["block"], v_rel, ops.K_TOKEN, case["bits_v"], case["v_block"], **stores["v"], **more)
    return {"stores": [stores for _, stores in s["layers"]], "orders": orders, "flags": s["flags"]}


def _prepare_harness(case, seed):
    dtype, ctx, hidden = DTYPES[case["dtype"]], case["ctx"], case["hidden"]
    heads = hidden // 128
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k, v = synth.synth_kv(1, heads, ctx, 128, seed=seed, dtype=dtype, device="cuda", apply_rope=True)
    codes = {}
    for which, x, bits in (("k", k, case["bits_k"]), ("v", v, case["bits_v"])):
        got = ops.quantize(x, 64, synth.rel_for_bits(bits), ops.K_TOKEN, bits=bits)
        codes[which] = (got.codes[0].cpu(), got.zero.flatten(), got.scale.flatten())
    q = _rows(gen, heads, 128, dtype=dtype)
    lanes = q.view(heads, 32, 4)
    q_lanes = torch.cat([lanes[:, :, :2].reshape(heads, -1), lanes[:, :, 2:].reshape(heads, -1)], dim=1).contiguous()
    w = torch.randn(heads, ctx, generator=gen, device="cuda").pow(2).softmax(dim=1).to(dtype)
    return dict(case=case, codes=codes, q=q, q_lanes=q_lanes, w=w, w_scaled=(w * codes["v"][2].unsqueeze(0)).contiguous())


def _run_harness(s):
    ctx, hidden, dtype = s["case"]["ctx"], s["case"]["hidden"], DTYPES[s["case"]["dtype"]]
    heads, out = hidden // 128, {}
    for which, cb, hb in (("k", 64, 128), ("v", 128, 64)):
        bits = s["case"]["bits_" + which]
        codes, zero, scale = s["codes"][which]
        info = torch.zeros((ctx // cb) * (hidden // hb), 2, dtype=U32)
        packed, back = torch.zeros_like(codes), torch.zeros_like(codes)
        size = getattr(packkv_cuda, which + "_encode_cpu")(codes, packed, info, ctx, hidden, cb, hb, bits)
        getattr(packkv_cuda, which + "_decode_cpu")(packed, info, back, ctx, hidden, cb, hb, bits)
        packed_dev, info_dev = packed.cuda(), info.cuda()
        if which == "k":
            product = torch.zeros(heads, ctx, dtype=dtype, device="cuda")
            packkv_cuda.kq_mat_vec_mul(packed_dev, info_dev, s["q_lanes"], product, ctx, hidden, cb, hb, bits)
            result = torch.empty_like(product)
            packkv_cuda.fused_kq(result, s["q"], zero, scale, product)
        else:
            product = torch.zeros(heads, 128, dtype=torch.float32, device="cuda")
            packkv_cuda.wv_mat_vec_mul(packed_dev, info_dev, s["w_scaled"], product, ctx, hidden, cb, hb, bits)
            product = product.to(dtype)
            result = torch.empty_like(product)
            packkv_cuda.fused_wv(result, s["w"], zero, scale, product)
        out[which] = [size, packed, info.view(torch.int32), back, product, result]
    return out


def prepare(case, seed):
    return {"kind": case["kind"],
            "state": {"decode": _prepare_decode, "session": _prepare_session, "encode": _prepare_encode, "harness": _prepare_harness}[case["kind"]](case, seed)}


def run(state):
    return {"decode": _run_decode, "session": _run_session, "encode": _run_encode, "harness": _run_harness}[state["kind"]](state["state"])


# ---- what a pass cannot do without --------------------------------------------------------------------------------------
def _packed(codes, bits):
    """Bytes of `codes` codes as packs of 16: the words at full width, a minimum and a length for each."""
    return codes * (bits + (bits + (3 if bits == 4 else 2)) / 16) / 8


def _params(batch, kv_heads, tokens, block, channel):
    return 4 * batch * (kv_heads * (tokens // block) * 128 if channel else tokens)


def work(case):
    if case["kind"] == "decode":
        B, H, G = case["batch"], case["kv_heads"], case["group"]
        n_comp, n_res = _split(case["ctx"], max(case["block"], case["v_block"]))
        codes = B * H * n_comp * 128
        one = _packed(codes, case["bits_k"]) + _packed(codes, case["bits_v"])
        one += _params(B, H, n_comp, case["block"], case["k_quant"] == "channel") + _params(B, H, n_comp, case["block"], False)
        one += 2 * B * H * n_res * 256 + 2 * B * H * G * 256
        return {"bytes": case["layers"] * one, "flops": case["layers"] * 4 * B * H * G * case["ctx"] * 128}
    if case["kind"] == "session":
        B, H, D, S, N, L = (case[x] for x in ("batch", "kv_heads", "head_dim", "prompt", "new_tokens", "layers"))
        bits = {x: cache.bits_for_rel(case[x + "_rel"]) for x in "kv"}
        # the prompt read, returned dense (K after RoPE) and packed
        n = 2 * L * B * H * S * D * 4 + sum(_packed(L * B * H * _split(S, case["block"])[0] * 128, b) for b in bits.values())
        for t in range(S + 1, S + N + 1):
            n_comp, n_res = _split(t, case["block"])
            n += L * B * H * ((sum(_packed(n_comp * 128, b) for b in bits.values()) + 4 * n_res * D) + (4 * t * D if case["materialize"] else 4 * case["group"] * D))
        return {"bytes": n, "flops": 0 if case["materialize"] else L * 4 * B * H * case["group"] * D * N * (S + N / 2)}
    if case["kind"] == "encode":
        B, H, S = case["batch"], case["kv_heads"], case["tokens"]
        codes = B * H * S * 128
        one = 4 * codes + _packed(codes, case["bits_k"]) + _packed(codes, case["bits_v"])
        one += _params(B, H, S, case["block"], case["k_quant"] == "channel") + _params(B, H, S, case["block"], False)
        return {"bytes": case["layers"] * one, "flops": 0}
    codes = case["ctx"] * case["hidden"]
    return {"bytes": sum(2 * codes + 4 * _packed(codes, case["bits_" + x]) for x in "kv") + 4 * 2 * case["ctx"] * (case["hidden"] // 128), "flops": 4 * codes}


def tolerance(case):
    if case["kind"] == "encode" or (case["kind"] == "session" and case["materialize"]):
        return "exact"           # codes, parameters and streams, and the dense view of them, are defined to the bit
    # scores, probabilities and outputs are rounded to the element type
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
