"""GPU: what the native host path (csrc/host.cpp) does before a kernel is launched.  The library's functions are replaced by a
stub for these tests, so nothing runs on the device: a call that the checks let through returns, one that they refuse raises."""
import ctypes

import pytest
import torch

from packkv_b200 import _lib, ops

pytestmark = pytest.mark.gpu

B, H, G, R = 3, 2, 2, 192
DTYPE = torch.float16


@pytest.fixture
def stubbed(cuda_device):
    """Every library function bound to CPython's PyGILState_Check: 0 (PKV_OK) where the caller has let go of the interpreter
    lock, 1 (a bad argument) where it has not."""
    host = _lib.host()
    stub = ctypes.cast(ctypes.pythonapi.PyGILState_Check, ctypes.c_void_p).value
    host.bind(*[stub] * len(_lib._HOST_FUNCTIONS))
    yield cuda_device
    _lib._host = None
    _lib.host()


def _empty(*shape, dtype=DTYPE, device="cuda"):
    return torch.zeros(*shape, dtype=dtype, device=device)


def test_no_call_holds_the_interpreter_lock(stubbed):
    """A launch may wait for room in the stream's queue, and a host callback that needs the lock may be what it waits for."""
    x, res = _empty(B, H, 1, 128), _empty(B, H, R, 128)
    ops.rope(x, _empty(1, 1, 128), _empty(1, 1, 128))
    ops.append_residual(x, x, res, res, 0)
    ops.widen_rows(_empty(B, H, 1, 96), None, res, None)
    ops.value_median_order(_empty(B, H, 64, 128), 64, 0.1)
    ops.decode_attention(_empty(B, H * G, 128), None, res, res, 1)



def test_append_and_plan_take_any_sequence(stubbed):
    q, res, new, cs = _empty(B, H * G, 128), _empty(B, H, R, 128), _empty(B, H, 1, 128), _empty(1, 1, 128)
    for append in ((new, new, cs, cs), [new, new, cs, cs], iter((new, new, None, None))):
        ops.decode_attention(q, None, res, res, 1, append=append)
    for plan in ((0, 0, 1), [0, 0, 1, 0], (0, 0, 1, 0, 7)):
        ops.decode_attention(q, None, res, res, 1, plan=plan)
    for append in ((new, new, cs), (new, new, cs, cs, cs), 3):
        with pytest.raises((ValueError, TypeError)):
            ops.decode_attention(q, None, res, res, 1, append=append)
    with pytest.raises(ValueError):
        ops.decode_attention(q, None, res, res, 1, plan=(0, 0))
