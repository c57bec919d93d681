"""The attention planner's choices, asked through pkv_attention_plan, which launches nothing and needs no GPU."""
import ctypes

import pytest

from packkv_b200 import _lib


def _plan(sequences, kv_heads, n_comp, n_res, group=4, bits=4, scratch=32 << 20):
    a = _lib.AttnArgs()
    for name in ("q", "out", "k_stream", "k_info", "k_scale", "k_zero", "v_stream", "v_info", "v_scale", "v_zero", "k_res", "v_res", "flags"):
        setattr(a, name, 1 << 28)                                   # an aligned address: sizes are looked at, memory is not
    a.k_capacity = a.v_capacity = 1 << 24
    a.param_tokens, a.param_blocks = n_comp, n_comp // 64
    a.n_comp, a.n_res, a.batch, a.kv_heads, a.group = n_comp, n_res, sequences, kv_heads, group
    a.cbk = a.cbv = 64
    a.bits_k = a.bits_v = bits
    a.scaling = 0.1
    plan = _lib.AttnPlan()
    assert _lib.lib().pkv_attention_plan(ctypes.byref(a), ctypes.byref(plan), scratch, 0) == _lib.PKV_OK
    return plan.cluster, plan.nsplit, plan.launches, plan.extra


@pytest.mark.parametrize("sequences,n_comp,n_res,cluster", [
    (18, 448, 152, 2), (14, 448, 152, 4), (16, 448, 152, 4), (18, 256, 164, 2),       # seven tiles to three CTAs, four to three: not there
    (18, 384, 137, 3), (14, 320, 150, 3), (14, 256, 164, 4), (1, 512, 188, 11),       # two tiles to each of three, idle SMs: as before
])
def test_teams_on_busy_gpus(sequences, n_comp, n_res, cluster):
    """8 KV heads: the cluster size that measured fastest among 2, 3 and 4 where an SM holds three teams of four warps or more."""
    assert _plan(sequences, 8, n_comp, n_res) == (cluster, 1, 1, 0)
