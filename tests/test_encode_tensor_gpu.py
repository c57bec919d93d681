"""GPU: the one-call encoder (pkv_encode_tensor: fp16/bf16 -> streams).  For K per-channel and V
per-token it runs the single-pass kernels; everything it writes -- streams, block tables, byte
counts, scales, zero-points -- must equal the CPU oracle (reference quantiser + reference codec)
bit for bit, for every bit width and block size, and must equal the two-stage GPU pipeline."""
import numpy as np
import pytest
import torch

from oracle import codec
from oracle import quant as Q
from packkv_b200 import encode, ops, synth

pytestmark = pytest.mark.gpu


def _bufs(B, H, S, cb, bits, which, mode, dtype, dev, extra_tokens=0):
    cap = S + extra_tokens
    shape = (B, H, cap // cb, 128) if mode == ops.K_CHANNEL else (B, cap)
    return dict(scale=torch.zeros(shape, dtype=dtype, device=dev), zero=torch.zeros(shape, dtype=dtype, device=dev),
                stream=torch.zeros(B, encode.stream_capacity(which, cap, H, cb, bits), dtype=torch.uint8, device=dev),
                info=torch.zeros(B, (cap // cb) * H * (1 if which == "k" else 2), 2, dtype=torch.int32, device=dev),
                stream_bytes=torch.zeros(B, dtype=torch.int32, device=dev), flags=ops.new_flags(dev))


def _oracle(x, which, mode, block, bits, hp):
    c, z, s = Q.quant_ints(x, block, synth.rel_for_bits(bits), "channel" if mode == ops.K_CHANNEL else "token", hp)
    codes = c.flatten(2, 3).permute(0, 2, 1, 3).flatten(2, 3).contiguous().to(torch.uint8)
    R = codec.restated()
    return [R.encode(which, codes[b].numpy(), block, bits) for b in range(x.shape[0])], z, s


@pytest.mark.parametrize("which,mode", [("k", ops.K_CHANNEL), ("v", ops.K_TOKEN), ("k", ops.K_TOKEN)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_encode_tensor_matches_oracle(cuda_device, which, mode, dtype):
    dev = cuda_device
    B, H = 2, 4
    k, v = synth.synth_kv(B, H, 384, 128, seed=41, dtype=dtype, apply_rope=True)
    x = k if which == "k" else v
    for bits in (2, 3, 4):
        for block in (32, 64, 128):
            for hp in (False, True):
                if hp and (bits, block) != (4, 64):
                    continue
                want, z, s = _oracle(x, which, mode, block, bits, hp)
                bufs = _bufs(B, H, 384, block, bits, which, mode, dtype, dev)
                ops.encode_tensor(which, x.to(dev), block, synth.rel_for_bits(bits), mode, bits, block, high_precision_zero=hp, **bufs)
                torch.cuda.synchronize()
                assert int(bufs["flags"].item()) == 0
                for b in range(B):
                    ws, wi = want[b]
                    assert int(bufs["stream_bytes"][b].item()) == ws.size, (bits, block)
                    assert np.array_equal(bufs["stream"][b, : ws.size].cpu().numpy(), ws), (bits, block, hp)
                    assert np.array_equal(bufs["info"][b].cpu().numpy().view(np.uint32), wi)
                shape = bufs["scale"].shape
                assert torch.equal(bufs["scale"].cpu().view(torch.int16), s.reshape(shape).contiguous().view(torch.int16))
                assert torch.equal(bufs["zero"].cpu().view(torch.int16), z.reshape(shape).contiguous().view(torch.int16))


def test_append_in_pieces_equals_one_call_and_flags(cuda_device):
    dev, dtype = cuda_device, torch.float16
    B, H, S = 3, 8, 512
    k, v = synth.synth_kv(B, H, S, 128, seed=43, dtype=dtype, device=dev)
    for which, mode, x in (("k", ops.K_CHANNEL, k), ("v", ops.K_TOKEN, v)):
        one = _bufs(B, H, S, 64, 4, which, mode, dtype, dev)
        ops.encode_tensor(which, x, 64, 1 / 14, mode, 4, 64, **one)
        parts = _bufs(B, H, S, 64, 4, which, mode, dtype, dev)
        for t0, t1 in ((0, 192), (192, 256), (256, 512)):
            ops.encode_tensor(which, x[:, :, t0:t1], 64, 1 / 14, mode, 4, 64, first_token=t0, **parts)
        torch.cuda.synchronize()
        for key in ("scale", "zero", "info", "stream_bytes"):
            assert torch.equal(one[key], parts[key]), key
        for b in range(B):
            n = int(one["stream_bytes"][b].item())
            assert torch.equal(one["stream"][b, :n], parts["stream"][b, :n])
    # codes that do not fit the bit width are reported, a stream that is too small is reported
    bufs = _bufs(B, H, S, 64, 3, "k", ops.K_CHANNEL, dtype, dev)
    ops.encode_tensor("k", k, 64, 0.1, ops.K_CHANNEL, 3, 64, **bufs)
    small = _bufs(B, H, S, 64, 4, "k", ops.K_CHANNEL, dtype, dev)
    small["stream"] = torch.zeros(B, 4096, dtype=torch.uint8, device=dev)
    ops.encode_tensor("k", k, 64, 1 / 14, ops.K_CHANNEL, 4, 64, **small)
    torch.cuda.synchronize()
    assert int(bufs["flags"].item()) & 2 and int(small["flags"].item()) & 1


@pytest.mark.parametrize("layout", ["bshd", "sliced", "padded_heads"])
@pytest.mark.parametrize("which,mode", [("k", ops.K_CHANNEL), ("k", ops.K_TOKEN), ("v", ops.K_TOKEN)])
def test_strided_inputs(cuda_device, layout, which, mode):
    """Inputs that are views of larger or differently ordered buffers (token-major memory, a window of a
    longer sequence, a subset of heads): same bytes as for the contiguous tensor."""
    dev, dtype = cuda_device, torch.bfloat16
    B, H, S, cb, bits = 2, 3, 192, 64, 4
    k, v = synth.synth_kv(B, H, S, 128, seed=47, dtype=dtype, apply_rope=True)
    x = (k if which == "k" else v).to(dev)
    if layout == "bshd":
        xs = x.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
    elif layout == "sliced":
        big = torch.zeros(B, H, S + 2 * cb, 128, dtype=dtype, device=dev)
        big[:, :, cb:cb + S] = x
        xs = big[:, :, cb:cb + S]
    else:
        big = torch.zeros(B, H + 2, S, 128, dtype=dtype, device=dev)
        big[:, 1:H + 1] = x
        xs = big[:, 1:H + 1]
    assert not xs.is_contiguous() and torch.equal(xs, x)
    rel = synth.rel_for_bits(bits)
    a, b = _bufs(B, H, S, cb, bits, which, mode, dtype, dev), _bufs(B, H, S, cb, bits, which, mode, dtype, dev)
    ops.encode_tensor(which, x, cb, rel, mode, bits, cb, **a)
    ops.encode_tensor(which, xs, cb, rel, mode, bits, cb, **b)
    torch.cuda.synchronize()
    assert int(a["flags"].item()) == 0 and int(b["flags"].item()) == 0
    for name in ("stream", "info", "stream_bytes", "scale", "zero"):
        assert torch.equal(a[name].view(torch.uint8), b[name].view(torch.uint8)), name


@pytest.mark.parametrize("which,mode", [("k", ops.K_CHANNEL), ("v", ops.K_TOKEN), ("k", ops.K_TOKEN)])
@pytest.mark.parametrize("H,S", [(3, 128), (12, 128), (1, 64), (2, 64 * 150)])
def test_direct_and_slot_forms(cuda_device, which, mode, H, S):
    """The encoder writes blocks straight to the stream after a look-back over the CTAs before it in the sequence;
    with more than 8 heads the per-token kernels go through slots and a compaction pass instead.  Head counts
    that leave the last CTA of a sequence partly empty (3), that take the slot form (12), the smallest input, and
    a sequence long enough for look-backs of more than one 32-entry window (150 token blocks, 75 K CTAs of 4
    blocks): all byte-exact against the oracle, three sequences so that chains of different sequences interleave."""
    dev, dtype = cuda_device, torch.float16
    B, block, bits = 3, 64, 4
    k, v = synth.synth_kv(B, H, S, 128, seed=43, dtype=dtype, apply_rope=True)
    x = k if which == "k" else v
    want, z, s = _oracle(x, which, mode, block, bits, False)
    bufs = _bufs(B, H, S, block, bits, which, mode, dtype, dev)
    for _ in range(2):   # a second call on the same scratch-free interface must start from clean look-back state
        ops.encode_tensor(which, x.to(dev), block, synth.rel_for_bits(bits), mode, bits, block, **bufs)
    torch.cuda.synchronize()
    assert int(bufs["flags"].item()) == 0
    for b in range(B):
        ws, wi = want[b]
        assert int(bufs["stream_bytes"][b].item()) == ws.size
        assert np.array_equal(bufs["stream"][b, : ws.size].cpu().numpy(), ws)
        assert np.array_equal(bufs["info"][b].cpu().numpy().view(np.uint32), wi)


@pytest.mark.parametrize("which,mode", [("k", ops.K_CHANNEL), ("v", ops.K_TOKEN), ("k", ops.K_TOKEN)])
@pytest.mark.parametrize("H,S,block,bits", [(8, 64, 64, 4), (5, 128, 64, 3), (8, 64 * 60, 64, 2), (8, 32, 32, 4), (7, 256, 128, 4), (6, 128, 128, 2)])
def test_launch_forms_by_size(cuda_device, which, mode, H, S, block, bits):
    """Sequences of one CTA (no look-back: one token block, or at most eight K blocks), V launches of few CTAs (16 warps
    each) and of more than the GPU has SMs (8 warps), in one call and behind tokens that are already there."""
    dev, dtype, B = cuda_device, torch.bfloat16, 3
    rel = synth.rel_for_bits(bits)
    k, v = synth.synth_kv(B, H, 2 * S, 128, seed=51, dtype=dtype, apply_rope=True)
    x = k if which == "k" else v
    want, z, s = _oracle(x, which, mode, block, bits, False)
    bufs = _bufs(B, H, 2 * S, block, bits, which, mode, dtype, dev)
    for t0 in (0, S):
        ops.encode_tensor(which, x[:, :, t0:t0 + S].to(dev), block, rel, mode, bits, block, first_token=t0, **bufs)
    torch.cuda.synchronize()
    assert int(bufs["flags"].item()) == 0
    for b in range(B):
        ws, wi = want[b]
        assert int(bufs["stream_bytes"][b].item()) == ws.size
        assert np.array_equal(bufs["stream"][b, : ws.size].cpu().numpy(), ws)
        assert np.array_equal(bufs["info"][b].cpu().numpy().view(np.uint32), wi)
    assert torch.equal(bufs["scale"].cpu().view(torch.int16), s.reshape(bufs["scale"].shape).contiguous().view(torch.int16))
    assert torch.equal(bufs["zero"].cpu().view(torch.int16), z.reshape(bufs["zero"].shape).contiguous().view(torch.int16))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("which,mode", [("k", ops.K_CHANNEL), ("v", ops.K_TOKEN), ("k", ops.K_TOKEN)])
@pytest.mark.parametrize("values", ["synthetic", "wide", "tiny", "special"])
def test_one_block_of_every_sequence(cuda_device, which, mode, dtype, values):
    """A call of one token block per sequence (a cluster of one-head CTAs) writes what a call of two blocks does: every block size and bit
    width, 1 to 8 heads, rows in any strides and through an order, parameters outside of the half-precision domain and without valid
    codes, the flags among the outputs; and a stream that is too small is flagged."""
    dev, gen = cuda_device, torch.Generator(device=cuda_device).manual_seed(7)
    for cb, bits, H in ((32, 4, 3), (64, 4, 8), (64, 3, 1), (64, 2, 5), (128, 4, 8), (128, 2, 2)):
        B, S = 3, 2 * cb
        x = torch.randn(B, S, H, 128, generator=gen, device=dev)
        if values == "wide":
            x = x * 900 + 3000
        elif values == "tiny":
            x = x * 1e-6
        elif values == "special":
            x[0, 3] = 0.0
            x[1, 5, 0, 7] = float("nan")
            x[1, cb + 1] = float("nan")
            x[2, 9, H - 1, 100] = float("inf")
            x[2, 2] = -0.0
        x = x.to(dtype).transpose(1, 2)                             # (B, H, S, 128), token-major in memory
        rel = synth.rel_for_bits(bits)
        order = None
        if cb == 64 and bits == 4:
            order = torch.stack([torch.randperm(cb, generator=torch.Generator().manual_seed(i)) for i in range(2 * B)]).view(B, 2, cb).to(torch.uint8).to(dev)
        two, one = (_bufs(B, H, S, cb, bits, which, mode, dtype, dev) for _ in range(2))
        ops.encode_tensor(which, x, cb, rel, mode, bits, cb, **two, **({} if order is None else dict(order=order, order_block=cb)))
        for i in range(2):
            ops.encode_tensor(which, x[:, :, i * cb: (i + 1) * cb], cb, rel, mode, bits, cb, first_token=i * cb, **one,
                              **({} if order is None else dict(order=order[:, i].contiguous(), order_block=cb)))
        for name in two:
            assert torch.equal(one[name].view(torch.uint8), two[name].view(torch.uint8)), (cb, bits, H, name)
        if values == "synthetic":
            assert int(one["flags"].item()) == 0
            small = _bufs(B, H, S, cb, bits, which, mode, dtype, dev)
            small["stream"] = torch.zeros(B, 256, dtype=torch.uint8, device=dev)
            ops.encode_tensor(which, x[:, :, :cb], cb, rel, mode, bits, cb, **small, **({} if order is None else dict(order=order[:, 0].contiguous(), order_block=cb)))
            assert int(small["flags"].item()) == 1 and torch.equal(small["info"][:, : one["info"].shape[1] // 2], one["info"][:, : one["info"].shape[1] // 2])


@pytest.mark.parametrize("cb,bits", [(64, 4), (64, 3), (32, 2)])
def test_v_forms_write_the_same(cuda_device, cb, bits):
    """V CTAs of 8 and of 16 warps, by the number of token blocks a call has (64-token blocks: up to 148 16 warps, one CTA to an SM; 200: 16, two to an SM;
    360 and 444: 8, three to an SM; 504: 8, four to an SM): the sequences of one call equal the same sequences in calls of one sequence each."""
    dev, dtype, H, rel = cuda_device, torch.float16, 8, synth.rel_for_bits(bits)
    for B, blocks in ((4, 126), (6, 60), (2, 100), (37, 12)):           # 504, 360, 200 and 444 token blocks
        _, v = synth.synth_kv(B, H, blocks * cb, 128, seed=B, dtype=dtype, device=dev)
        all_ = _bufs(B, H, blocks * cb, cb, bits, "v", ops.K_TOKEN, dtype, dev)
        ops.encode_tensor("v", v, cb, rel, ops.K_TOKEN, bits, cb, **all_)
        assert int(all_["flags"].item()) == 0
        for b in (0, B - 1):
            one = _bufs(1, H, blocks * cb, cb, bits, "v", ops.K_TOKEN, dtype, dev)
            ops.encode_tensor("v", v[b: b + 1], cb, rel, ops.K_TOKEN, bits, cb, **one)
            for name in ("scale", "zero", "stream", "info", "stream_bytes"):
                assert torch.equal(one[name][0], all_[name][b]), (B, b, name)


@pytest.mark.parametrize("which,mode", [("k", ops.K_CHANNEL), ("v", ops.K_TOKEN), ("k", ops.K_TOKEN)])
@pytest.mark.parametrize("cb", [32, 64, 128])
def test_one_block_at_the_limits_of_the_form(cuda_device, which, mode, cb):
    """Calls of one token block per sequence around the numbers of one-head CTAs up to which a cluster takes a sequence, every number of heads:
    both forms write what a call of two blocks per sequence does."""
    dev, dtype, rel = cuda_device, torch.bfloat16, synth.rel_for_bits(3)
    for H in range(1, 9):
        for ctas in (444, 518, 592) if cb == 32 else (592,):
            for B in (ctas // H, ctas // H + 1):
                x = torch.randn(B, H, 2 * cb, 128, generator=torch.Generator(device=dev).manual_seed(B), device=dev).to(dtype)
                two, one = (_bufs(B, H, 2 * cb, cb, 3, which, mode, dtype, dev) for _ in range(2))
                ops.encode_tensor(which, x, cb, rel, mode, 3, cb, **two)
                for i in range(2):
                    ops.encode_tensor(which, x[:, :, i * cb: (i + 1) * cb], cb, rel, mode, 3, cb, first_token=i * cb, **one)
                for name in two:
                    assert torch.equal(one[name].view(torch.uint8), two[name].view(torch.uint8)), (H, B, name)


@pytest.mark.parametrize("heads,cb,bits,ordered", [(5, 64, 4, True), (6, 32, 3, False), (9, 64, 2, False), (16, 64, 4, True), (16, 32, 4, False), (8, 128, 4, False),
                                                   (5, 128, 2, True)])
def test_v_forms_of_other_heads_and_blocks(cuda_device, heads, cb, bits, ordered):
    """The forms of the V launch for other numbers of heads, 128-token blocks, bf16 and rows read through an order write the same; numbers of token
    blocks on both sides of each line between them: 148, 296, 444, 592 and 888."""
    dev, dtype, rel = cuda_device, torch.bfloat16, synth.rel_for_bits(bits)
    g = torch.Generator(device=dev).manual_seed(1)
    for blocks in (148, 149, 296, 297, 444, 445, 592, 593, 889):
        v = torch.randn(1, blocks * cb, heads, 128, generator=g, device=dev).to(dtype).transpose(1, 2)
        order = torch.argsort(torch.rand(blocks, cb, generator=g, device=dev)).to(torch.uint8) if ordered else None
        more = lambda lo, hi: {} if order is None else dict(order=order[lo:hi].contiguous(), order_block=cb)
        all_, parts = (_bufs(1, heads, blocks * cb, cb, bits, "v", ops.K_TOKEN, dtype, dev) for _ in range(2))
        ops.encode_tensor("v", v, cb, rel, ops.K_TOKEN, bits, cb, **all_, **more(0, blocks))
        for lo in range(0, blocks, 100):                            # calls of up to 100 token blocks
            hi = min(blocks, lo + 100)
            ops.encode_tensor("v", v[:, :, lo * cb: hi * cb], cb, rel, ops.K_TOKEN, bits, cb, first_token=lo * cb, **parts, **more(lo, hi))
        for name in all_:
            assert torch.equal(all_[name].view(torch.uint8), parts[name].view(torch.uint8)), (blocks, name)


@pytest.mark.parametrize("heads,cb,bits", [(4, 64, 4), (1, 64, 3), (2, 128, 4), (4, 128, 3), (3, 32, 2)])
def test_v_forms_of_little_work(cuda_device, heads, cb, bits):
    """V launches of little work per CTA on both sides of the lines between their forms (148, 444, 592 and 888 token blocks), in blocks of every size:
    the calls' results equal those of calls of at most 100 token blocks."""
    dev, dtype, rel = cuda_device, torch.float16, synth.rel_for_bits(bits)
    g = torch.Generator(device=dev).manual_seed(2)
    for blocks in (148, 149, 444, 445, 592, 593, 888, 889):
        v = torch.randn(1, heads, blocks * cb, 128, generator=g, device=dev).to(dtype)
        all_, parts = (_bufs(1, heads, blocks * cb, cb, bits, "v", ops.K_TOKEN, dtype, dev) for _ in range(2))
        ops.encode_tensor("v", v, cb, rel, ops.K_TOKEN, bits, cb, **all_)
        for lo in range(0, blocks, 100):
            hi = min(blocks, lo + 100)
            ops.encode_tensor("v", v[:, :, lo * cb: hi * cb], cb, rel, ops.K_TOKEN, bits, cb, first_token=lo * cb, **parts)
        assert int(all_["flags"].item()) == 0
        for name in all_:
            assert torch.equal(all_[name].view(torch.uint8), parts[name].view(torch.uint8)), (blocks, name)


@pytest.mark.parametrize("heads,cb,bits,blocks", [(4, 64, 4, (666, 667, 962, 963, 1184, 1185, 1332, 1333)), (6, 64, 4, (592, 593, 666, 667)), (6, 64, 2, (592, 593)),
                                                  (10, 64, 4, (296, 297, 444, 445, 592, 593)), (13, 32, 3, (148, 149)), (8, 32, 4, (888, 889)),
                                                  (3, 128, 3, (296, 297, 888, 889, 1184, 1185)), (2, 128, 4, (1332, 1333)), (10, 128, 2, (148, 149, 296, 297, 444, 445)), (8, 128, 2, (74, 75, 126, 128, 148, 149, 296, 297)),
                                                  (4, 128, 4, (74, 75, 296, 297))])
def test_v_blocks_through_a_tile_and_from_registers(cuda_device, heads, cb, bits, blocks):
    """V launches on both sides of the lines at which the way of a block changes, in calls of several sequences, blocks of every conversion among
    them: the calls' results equal those of calls of at most 60 token blocks of one sequence."""
    dev, dtype, rel = cuda_device, torch.bfloat16, synth.rel_for_bits(bits)
    g = torch.Generator(device=dev).manual_seed(3)
    for n in blocks:
        B = next(B for B in (3, 2, 1) if n % B == 0)
        v = torch.randn(B, n // B * cb, heads, 128, generator=g, device=dev).to(dtype).transpose(1, 2)
        for i, (spread, middle) in enumerate(((8, 1000), (8, 8000), (3e4, 0))):      # zero-points that the faster conversions do not take
            at = slice((5 + i) * cb, (6 + i) * cb)
            v[0, :, at] = (v[0, :, at].float() * spread + middle).to(dtype)
        all_ = _bufs(B, heads, n // B * cb, cb, bits, "v", ops.K_TOKEN, dtype, dev)
        ops.encode_tensor("v", v, cb, rel, ops.K_TOKEN, bits, cb, **all_)
        for b in range(B):
            one = _bufs(1, heads, n // B * cb, cb, bits, "v", ops.K_TOKEN, dtype, dev)
            for lo in range(0, n // B, 60):
                hi = min(n // B, lo + 60)
                ops.encode_tensor("v", v[b: b + 1, :, lo * cb: hi * cb], cb, rel, ops.K_TOKEN, bits, cb, first_token=lo * cb, **one)
            for name in ("scale", "zero", "stream", "info", "stream_bytes"):
                assert torch.equal(one[name].view(torch.uint8), all_[name][b: b + 1].view(torch.uint8)), (n, b, name)
