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



def _accepted_and_refused(call, good, bad):
    for change in good:
        call(**change)
    for change in bad:
        with pytest.raises(ValueError):
            call(**change)


def test_attention_checks_what_the_kernel_indexes(stubbed):
    q, res = _empty(B, H * G, 128), _empty(B, H, R, 128)
    big = _empty(B + 1, H + 1, R + 64, 128)

    def call(k=res, v=res, n_res=R, **more):
        ops.decode_attention(q, None, k, v, n_res, kv_heads=H, **more)

    _accepted_and_refused(
        call,
        [dict(), dict(k=big, v=big), dict(k=big[:B, :H], v=big[:B, :H]), dict(out=torch.empty_like(q)), dict(out=_empty(B, 1, H * G * 128)),
         dict(flags=_empty(2, dtype=torch.int32)), dict(flags=_empty(1, dtype=torch.int64))],
        [dict(n_res=R + 1),                                                   # more rows than the residual has
         dict(k=res[: B - 1], v=res[: B - 1]), dict(k=res[:, : H - 1], v=res[:, : H - 1]),
         dict(v=res[:1]), dict(v=res[:, :1]), dict(v=res[:, :, : R - 1]),     # V with K's strides, not its sizes
         dict(k=_empty(B, H, R, 64).as_strided((B, H, R // 2, 64), (H * R * 64, R * 64, 128, 1)), v=res, n_res=1),
         dict(out=_empty(B, H * G - 1, 128)), dict(out=_empty(B, H * G, 128, dtype=torch.float32)), dict(out=_empty(B, H * G, 256)[..., :128]),
         dict(flags=_empty(0, dtype=torch.int32)), dict(flags=_empty(1, dtype=torch.uint8))])
    new = _empty(B, H, 1, 128)

    def append(cos):
        call(append=(new, new, cos, cos))

    _accepted_and_refused(append, [dict(cos=_empty(n, 1, 128)) for n in (1, B, B + 1)] + [dict(cos=_empty(1, 128))],
                          [dict(cos=_empty(B - 1, 1, 128)), dict(cos=_empty(B, 2, 128))])


@pytest.mark.parametrize("which,mode", [("k", ops.K_CHANNEL), ("k", ops.K_TOKEN), ("v", ops.K_TOKEN)])
def test_encoder_checks_what_it_writes(stubbed, which, mode):
    S, first, block = 128, 64, 64
    x, per = _empty(B, H, S, 128), H if which == "k" else 2 * H
    rows = (first + S) // block * per

    def params(b=B, h=H, tokens=first + S, dtype=DTYPE):
        return _empty(*((b, h, tokens // block, 128) if mode == ops.K_CHANNEL else (b, tokens)), dtype=dtype)

    base = dict(scale=params(), zero=params(), stream=_empty(B, 1 << 16, dtype=torch.uint8), info=_empty(B, rows, 2, dtype=torch.int32),
                stream_bytes=_empty(B, dtype=torch.int32), flags=_empty(1, dtype=torch.int32))

    def call(**change):
        ops.encode_tensor(which, x, block, 0.1, mode, 4, block, **{**base, "first_token": first, **change})

    larger = params(b=B + 1, tokens=4096)
    _accepted_and_refused(
        call,
        [dict(), dict(scale=larger, zero=larger), dict(stream=_empty(B + 1, 1 << 17, dtype=torch.uint8)[:, : 1 << 16]), dict(info=_empty(B, rows + 9, 2, dtype=torch.int32)),
         dict(stream_bytes=_empty(B + 1, dtype=torch.int32)), dict(first_token=0)],
        [dict(first_token=2 * first), dict(first_token=-block),
         dict(scale=params(b=B - 1)), dict(zero=params(b=B - 1)), dict(zero=params(tokens=S)), dict(scale=params(dtype=torch.bfloat16)),
         dict(scale=params(dtype=torch.float32)), dict(scale=larger[:, ..., ::2], zero=larger[:, ..., ::2]),
         dict(stream=_empty(B - 1, 1 << 16, dtype=torch.uint8)), dict(stream=_empty(B, 1 << 16, dtype=torch.int32)),
         dict(info=_empty(B, rows - 1, 2, dtype=torch.int32)), dict(info=_empty(B - 1, rows, 2, dtype=torch.int32)),
         dict(info=_empty(B, rows, 2, dtype=torch.int16)), dict(info=_empty(B, rows, 4, dtype=torch.int32)[..., :2]),
         dict(stream_bytes=_empty(B - 1, dtype=torch.int32)), dict(stream_bytes=_empty(B, dtype=torch.uint8)),
         dict(flags=_empty(0, dtype=torch.int32))])
    if mode == ops.K_CHANNEL:
        with pytest.raises(ValueError):
            call(scale=params(h=H - 1), zero=params(h=H - 1))
    with pytest.raises(RuntimeError, match="not supported"):
        ops.encode_tensor(which, x, block, 0.1, ops.Q_VECTOR, 4, block, **base)


def test_rows_check_what_they_read_and_write(stubbed):
    T, x, y = 5, _empty(B, H, 5, 128), _empty(B, H, 5, 96)
    res = _empty(B, H, R, 128)

    def append(k=res, cos=None):
        ops.append_residual(x, x, k, k, 0, cos, cos)

    def widen(k=res, cos=None):
        ops.widen_rows(y, y, k, k, 0, cos, cos)

    def rope(cos=_empty(1, 5, 128), out=None):
        ops.rope(x, cos, cos, out)

    for call, D in ((append, 128), (widen, 96), (rope, 128)):
        _accepted_and_refused(call, [dict(cos=_empty(n, T, D)) for n in (1, B, B + 1)] + [dict(cos=_empty(n, 1, T, D)) for n in (1, B)],
                              [dict(cos=_empty(B - 1, T, D)), dict(cos=_empty(T, D)), dict(cos=_empty(1, T + 1, D))])
    _accepted_and_refused(append, [dict(), dict(k=_empty(B + 1, H + 1, R, 128))],
                          [dict(k=_empty(B - 1, H, R, 128)), dict(k=_empty(B, H - 1, R, 128)), dict(k=_empty(B, H, R, 64).as_strided((B, H, R // 2, 64), (H * R * 64, R * 64, 128, 1)))])
    _accepted_and_refused(rope, [dict(out=_empty(B, 5, H, 128).transpose(1, 2)), dict(out=_empty(B, H, 9, 128))],
                          [dict(out=_empty(B, H, 4, 128)), dict(out=_empty(B, H, 5, 128, dtype=torch.float32)), dict(out=_empty(B, H, 128, 5).transpose(2, 3))])
    with pytest.raises(ValueError):
        ops.value_median_order(_empty(B, H, 64, 128), 64, 0.1, flags=_empty(0, dtype=torch.int32))
