"""The attention planner's choices, asked through pkv_attention_plan, which launches nothing and needs no GPU."""
import ctypes

import pytest

from packkv_b200 import _lib


def _ask(sequences, kv_heads, n_comp, n_res, group=4, bits=4, scratch=32 << 20, block=64, plan=(0, 0, 0), exchange=0):
    a = _lib.AttnArgs()
    for name in ("q", "out", "k_stream", "k_info", "k_scale", "k_zero", "v_stream", "v_info", "v_scale", "v_zero", "k_res", "v_res", "flags"):
        setattr(a, name, 1 << 28)                                   # an aligned address: sizes are looked at, memory is not
    a.k_capacity = a.v_capacity = 1 << 24
    a.param_tokens, a.param_blocks = n_comp, n_comp // block
    a.n_comp, a.n_res, a.batch, a.kv_heads, a.group = n_comp, n_res, sequences, kv_heads, group
    a.cbk = a.cbv = block
    a.bits_k = a.bits_v = bits
    a.scaling = 0.1
    plan, sends = _lib.AttnPlan(*plan), ctypes.c_int32(-1)
    again = _lib.AttnPlan(plan.cluster, plan.nsplit, plan.launches)
    assert _lib.lib().pkv_attention_plan(ctypes.byref(a), ctypes.byref(plan), scratch, exchange) == _lib.PKV_OK
    assert _lib.lib().pkv_attention_sends(ctypes.byref(a), ctypes.byref(again), scratch, exchange, ctypes.byref(sends)) == _lib.PKV_OK
    assert bytes(again) == bytes(plan)
    return (plan.cluster, plan.nsplit, plan.launches, plan.extra), sends.value


def _plan(*args, **more):
    return _ask(*args, **more)[0]


@pytest.mark.parametrize("sequences,n_comp,n_res,cluster", [
    (18, 448, 152, 2), (14, 448, 152, 4), (16, 448, 152, 4), (18, 256, 164, 2),       # seven tiles to three CTAs, four to three: not there
    (18, 384, 137, 3), (14, 320, 150, 3), (14, 256, 164, 4), (1, 512, 188, 11),       # two tiles to each of three, idle SMs: as before
])
def test_teams_on_busy_gpus(sequences, n_comp, n_res, cluster):
    """8 KV heads: the cluster size that measured fastest among 2, 3 and 4 where an SM holds three teams of four warps or more."""
    assert _plan(sequences, 8, n_comp, n_res) == (cluster, 1, 1, 0)


@pytest.mark.parametrize("sequences,group,n_comp,plan,sends", [
    (8, 7, 5120, (15, 1, 1), 0), (7, 7, 5120, (15, 1, 1), 1),         # two CTAs to an SM, one with the receive area: seven clusters of 15 fit then
    (8, 8, 5120, (15, 1, 1), 0), (7, 8, 5120, (15, 1, 1), 1),
    (8, 4, 8192, (4, 1, 1), 1), (8, 4, 16384, (4, 1, 1), 1),          # 512 and 1024 tokens to a warp
    (8, 4, 1024, (1, 1, 1), 0), (8, 4, 1024, (8, 1, 1), 1), (8, 4, 1024, (1, 3, 2), 0), (8, 4, 1024, (3, 3, 2), 1),     # clusters of one CTA send nothing
])
def test_sums_are_sent_where_the_receive_area_costs_no_wave(sequences, group, n_comp, plan, sends):
    """128-token blocks, one KV head: whether the cluster's CTAs send one another their sums."""
    assert _ask(sequences, 1, n_comp, 213, group, block=128, plan=plan) == ((*plan, 0), sends)


def test_launches_with_an_exchange_read_their_sums():
    assert _ask(1, 8, 512, 188, plan=(8, 1, 1))[1] == 1 and _ask(1, 8, 512, 188, plan=(8, 1, 1), exchange=1)[1] == 0
