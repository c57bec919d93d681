"""GPU: the dense view of a layer (pkv_dense) against the oracle's quantise -> dequantise on CPU, bit for bit: every
element is the result of the same two rounded operations."""
import pytest
import torch

from helpers import layer_from_oracle
from oracle import quant as Q
from packkv_b200 import encode, ops, synth
from packkv_b200.config import QuantMode, RepackMethod

pytestmark = pytest.mark.gpu


def _check(layer, kd, vd, k_res, v_res, n_res, dim, block, flags):
    for which, dense, res in (("k", kd, k_res), ("v", vd, v_res)):
        got = ops.dense(which, layer, res, n_res, dim, block, flags).cpu()
        want = torch.cat([dense[..., :dim], res[:, :, :n_res, :dim].cpu()], dim=2)
        assert got.shape == want.shape
        assert torch.equal(got.view(torch.int16), want.view(torch.int16)), which
    assert int(flags.item()) == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("k_mode", ["channel", "token"])
@pytest.mark.parametrize("bits,block,dim,n_res,hp", [(4, 64, 128, 133, False), (3, 64, 96, 1, False), (2, 128, 128, 0, False), (4, 128, 72, 16, True),
                                                     (3, 128, 64, 17, True)])
def test_dense_matches_the_oracle(cuda_device, dtype, k_mode, bits, block, dim, n_res, hp):
    dev = cuda_device
    B, H, S = 2, 3, 384
    k, v = synth.synth_kv(B, H, S, 128, seed=bits * 10 + block, dtype=dtype)
    k[0, 0, 16:32], v[1, 1, 16:32] = k[0, 0, 16:17], 0.01  # packs of width 0
    k[1, 2, 5] *= 300                                      # and one far outside the rest
    rel = synth.rel_for_bits(bits)
    layer, kd, vd = layer_from_oracle(k, v, block=block, bits_k=bits, bits_v=bits, k_mode=k_mode, cbk=block, cbv=block, rel_k=rel, rel_v=rel, device=dev, hp=hp)
    res = [torch.randn(B, H, 192, 128).to(dtype).to(dev) for _ in range(2)]
    _check(layer, kd, vd, *res, n_res, dim, block, ops.new_flags(dev))


@pytest.mark.parametrize("cbv", [64, 128])
def test_dense_returns_reordered_tokens_in_source_order(cuda_device, cbv):
    dev = cuda_device
    B, H, S = 2, 2, 256
    k, v = synth.synth_kv(B, H, S, 128, seed=3, dtype=torch.bfloat16)
    rel = synth.rel_for_bits(4)
    layer = encode.compress_kv(k.to(dev), v.to(dev), block=64, bits_k=4, bits_v=4, k_rel=rel, v_rel=rel, k_mode=QuantMode.ChannelQuant, cbk=64, cbv=cbv,
                               repack_method=RepackMethod.MEDIAN)
    assert not torch.equal(layer.order[0, 0].cpu(), torch.arange(64, dtype=torch.uint8))
    kd, vd = (Q.dequant(*Q.quant_ints(x, 64, rel, mode, False)) for x, mode in ((k, "channel"), (v, "token")))
    res = torch.zeros(B, H, 192, 128, dtype=torch.bfloat16, device=dev)
    _check(layer, kd, vd, res, res, 3, 128, 64, ops.new_flags(dev))


def test_dense_flags_blocks_outside_the_stream(cuda_device):
    dev = cuda_device
    k, v = synth.synth_kv(1, 2, 128, 128, seed=4, dtype=torch.float16)
    rel = synth.rel_for_bits(4)
    layer, kd, _ = layer_from_oracle(k, v, block=64, bits_k=4, bits_v=4, k_mode="channel", cbk=64, cbv=64, rel_k=rel, rel_v=rel, device=dev)
    layer.k_info[0, 1, 0] = layer.k_stream.shape[1]
    flags = ops.new_flags(dev)
    got = ops.dense("k", layer, None, 0, 128, 64, flags).cpu()
    assert int(flags.item()) == 4
    assert torch.equal(got[:, 0], kd[:, 0]) and torch.equal(got[:, 1, 64:], kd[:, 1, 64:])
    want = layer.k_zero[0, 1, 0].cpu() * layer.k_scale[0, 1, 0].cpu()             # codes 0
    assert torch.equal(got[0, 1, :64], want.expand(64, 128))


@pytest.mark.parametrize("cbv", [64, 128])
@pytest.mark.parametrize("entry", [255, 64, 7])
def test_dense_keeps_groups_that_are_no_permutation_in_stored_order(cuda_device, cbv, entry):
    """An entry outside its group, or one that is there twice, in the last group of the last sequence and in one before
    others: flagged, the group's rows in stored order, every other row and the residual untouched."""
    dev = cuda_device
    B, H, S, n_res = 2, 2, 256, 5
    k, v = synth.synth_kv(B, H, S, 128, seed=6, dtype=torch.float16, device=dev)
    rel = synth.rel_for_bits(4)
    layer = encode.compress_kv(k, v, block=64, bits_k=4, bits_v=4, k_rel=rel, v_rel=rel, cbk=64, cbv=cbv, repack_method=RepackMethod.MEDIAN)
    res = torch.randn(B, H, 192, 128, device=dev).half()
    want = {which: ops.dense(which, layer, res, n_res, 128, 64) for which in "kv"}
    broken = layer.order.clone()
    for b, g in ((0, 1), (B - 1, S // 64 - 1)):
        stored = layer.order[b, g].long() + 64 * g
        for which in "kv":
            want[which][b, :, 64 * g:64 * g + 64] = want[which][b][:, stored]
        row = int((broken[b, g] != entry).nonzero()[0])
        broken[b, g, row] = entry
    layer.order = broken
    for which in "kv":
        flags = ops.new_flags(dev)
        got = ops.dense(which, layer, res, n_res, 128, 64, flags)
        assert int(flags.item()) == 4
        assert torch.equal(got, want[which])


def test_dense_refuses_an_order_of_another_form(cuda_device):
    dev = cuda_device
    k, v = synth.synth_kv(1, 1, 128, 128, seed=7, dtype=torch.float16, device=dev)
    layer = encode.compress_kv(k, v, block=64, bits_k=4, bits_v=4, k_rel=1 / 14, v_rel=1 / 14, repack_method=RepackMethod.MEDIAN)
    order = layer.order
    for other in (order.int(), order[:, :1], order.view(1, 128), torch.zeros(1, 2, 128, dtype=torch.uint8, device=dev)[..., ::2]):
        layer.order = other
        with pytest.raises(ValueError):
            ops.dense("k", layer, None, 0, 128, 64)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("k_mode,block,cbk,cbv,S,repack", [
    ("channel", 64, 128, 128, 384, RepackMethod.NONE), ("channel", 128, 64, 64, 384, RepackMethod.NONE), ("channel", 32, 128, 64, 256, RepackMethod.NONE),
    ("token", 128, 64, 64, 256, RepackMethod.MEDIAN), ("token", 128, 64, 128, 256, RepackMethod.GREEDY), ("token", 64, 128, 128, 256, RepackMethod.MEDIAN)])
def test_dense_takes_quantisation_blocks_of_other_sizes_than_the_streams(cuda_device, dtype, k_mode, block, cbk, cbv, S, repack):
    """compress_kv stores such layers; a reorder block may span stream blocks, and parameters change inside one."""
    dev, B, H, rel = cuda_device, 2, 2, synth.rel_for_bits(4)
    k, v = synth.synth_kv(B, H, S, 128, seed=block + cbk, dtype=dtype)
    layer = encode.compress_kv(k.to(dev), v.to(dev), block=block, bits_k=4, bits_v=4, k_rel=rel, v_rel=rel, cbk=cbk, cbv=cbv, repack_method=repack,
                               k_mode=QuantMode.ChannelQuant if k_mode == "channel" else QuantMode.TokenQuant)
    res = torch.zeros(B, H, 192, 128, dtype=dtype, device=dev)
    flags = ops.new_flags(dev)
    for which, x, mode in (("k", k, k_mode), ("v", v, "token")):
        want = Q.dequant(*Q.quant_ints(x, block, rel, mode, False))
        got = ops.dense(which, layer, res, 0, 128, block, flags).cpu()
        assert torch.equal(got.view(torch.int16), want.view(torch.int16)), which
    assert int(flags.item()) == 0


def test_dense_of_per_token_layers_needs_no_whole_quantisation_block(cuda_device):
    dev, rel = cuda_device, synth.rel_for_bits(4)
    k, v = synth.synth_kv(1, 2, 192, 128, seed=9, dtype=torch.float16)
    layer = encode.compress_kv(k.to(dev), v.to(dev), block=64, bits_k=4, bits_v=4, k_rel=rel, v_rel=rel, k_mode=QuantMode.TokenQuant)
    for which, x in (("k", k), ("v", v)):
        want = Q.dequant(*Q.quant_ints(x, 64, rel, "token", False))
        assert torch.equal(ops.dense(which, layer, None, 0, 128, 128).cpu(), want)
