"""Buffers of the caller's are looked over before anything is launched: too short, of another type, in
pieces or on the host they are refused.  FakeTensors have a CUDA device and shapes but no memory, so the
checks run without a GPU, and a call that got past them could not launch."""

from types import SimpleNamespace

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from mosaicist_b200 import ops

BF16, F32, U8, I32 = torch.bfloat16, torch.float32, torch.uint8, torch.int32


def _t(*shape, dtype=BF16, device="cuda"):
    return torch.empty(shape, dtype=dtype, device=device)


def _bad(rows, cols, dtype, other):
    """Buffers that do not do for (rows, cols) of a type."""
    return [_t(rows - 1, cols, dtype=dtype), _t(rows, cols, dtype=other), _t(cols, rows, dtype=dtype).t(),
            _t(rows, cols, dtype=dtype, device="cpu")]


def _refused(call, *buffers):
    for b in buffers:
        with pytest.raises(ValueError):
            call(b)


@pytest.fixture(autouse=True)
def fake():
    with FakeTensorMode():
        yield


def test_int4_buffers():
    b_q, scales = _t(2, 256, 64, dtype=U8), _t(2, 256, 1)
    a, offs, rows = _t(256, 128), _t(2, dtype=I32), _t(2, dtype=I32)
    weights = [_t(2, 256, 127), _t(1, 256, 128), _t(2, 256, 128, dtype=torch.float16), _t(2, 128, 256).transpose(1, 2),
               _t(2, 256, 128, device="cpu")]
    _refused(lambda b: ops.dequant_int4(b_q, scales, out=b), *weights)
    _refused(lambda b: ops.mixed_grouped_gemm_int4(a, b_q, scales, offs, rows, workspace=b), *weights)
    _refused(lambda b: ops.mixed_grouped_gemm_int4(a, b_q, scales, offs, rows, out=b), *_bad(256, 256, BF16, F32))
    _refused(lambda b: ops.ragged_grouped_gemm_bf16(a, _t(2, 256, 128), offs, rows, out=b), *_bad(256, 256, BF16, F32))


@pytest.mark.parametrize("tiled,ragged", [(True, False), (False, False), (True, True)])
def test_mxfp8_buffers(tiled, ragged):
    x = _t(200, 128)
    kw = dict(group_offsets=_t(2, dtype=I32), group_rows=_t(2, dtype=I32)) if ragged else {}
    q, sf = _t(200, 128, dtype=U8), _t(2, 1, 32, 16, dtype=U8) if tiled else _t(200, 4, dtype=U8)
    _refused(lambda b: ops.quantize_mxfp8(x, tiled, out=(b, sf), **kw), *_bad(200, 128, U8, I32))
    _refused(lambda b: ops.quantize_mxfp8(x, tiled, out=(q, b), **kw), sf[:1].flatten()[:-1], sf.to(I32), sf.cpu())


def test_dense_out():
    a, b = _t(64, 128), _t(128, 256)
    _refused(lambda c: ops.gemm_f16(a, b, out=c), *_bad(64, 256, BF16, torch.float16))


def test_routed_layer_buffers():
    from mosaicist_b200.moe import _host_ops

    T, h, E, k = 16, 256, 8, 2
    i32 = lambda *s: _t(*s, dtype=I32)
    layer = SimpleNamespace(ids=i32(T, k), weights=_t(T, k, dtype=F32), rank=i32(T, k), group_rows=i32(E), group_offsets=i32(E),
                            total_rows=i32(1), scratch=i32(4), topk=k, E=E, expert_first=0, input_gs=_t(E, dtype=F32), h=h,
                            a_q=_t(1152, h // 2, dtype=U8), a_sf=_t(9, h // 64, 32, 16, dtype=U8), row_weight=_t(1152, dtype=F32),
                            row_token=i32(1152), sf_rows=None, rows_cap=1152, y=_t(1152, h))
    tokens, logits = _t(T, h), _t(T, E, dtype=F32)
    # (a call with fewer tokens than the layer was built for is a smaller call)
    _refused(lambda b: _host_ops.moe_dispatch(layer, b, logits), *_bad(T, h, BF16, F32)[1:], _t(T, h - 64), _t(T + 1, h))
    _refused(lambda b: _host_ops.moe_dispatch(layer, tokens, b), _t(T + 1, E, dtype=F32), _t(T, E), _t(E, T, dtype=F32).t(),
             _t(T, E, dtype=F32, device="cpu"))
    _refused(lambda b: _host_ops.moe_route(layer, b), _t(T + 1, E, dtype=F32), _t(T, E))
    _refused(lambda b: _host_ops.moe_combine(layer, tokens, b), *_bad(T, h, BF16, F32))


def test_layer_attributes_may_be_computed():
    """A buffer that only the attribute look-up itself holds stays alive for the call."""
    from mosaicist_b200.moe import _host_ops

    asked = []

    class Layer:
        topk = 2

        @property
        def ids(self):
            asked.append("ids")
            return _t(16, 2, dtype=I32)

        @property
        def weights(self):
            asked.append("weights")
            return _t(15, 2, dtype=F32)

    for _ in range(20):
        with pytest.raises(ValueError, match="weights holds 30 elements"):
            _host_ops.moe_route(Layer(), _t(16, 8, dtype=F32))
    assert asked[:2] == ["ids", "weights"]
    Layer.ids = None
    with pytest.raises(ValueError, match="missing"):
        _host_ops.moe_route(Layer(), _t(16, 8, dtype=F32))


def test_first_calls_from_several_threads():
    """The library's entry points are fetched by whichever threads call first: all of them get a whole
    table and none waits for another.  (In a process of its own: the table is fetched once.)"""
    import pathlib
    import subprocess
    import sys

    code = """
import threading, time, torch
from torch._subclasses.fake_tensor import FakeTensorMode
from mosaicist_b200 import _lib, ops
fetch, calls = _lib.addresses, []
def slow():
    calls.append(1)
    time.sleep(0.2)                  # other threads get the GIL here
    return fetch()
_lib.addresses = slow
with FakeTensorMode():
    a, b = (torch.empty(s, dtype=torch.bfloat16, device="cuda") for s in ((64, 128), (128, 64)))
    out = torch.empty((64, 64), dtype=torch.bfloat16, device="cuda")
seen = []
def call():
    try:
        ops.gemm_f16(a, b, out=out)  # no memory behind the tensors: refused by torch or the library
    except RuntimeError as e:
        seen.append(str(e))
threads = [threading.Thread(target=call) for _ in range(8)]
[t.start() for t in threads]
[t.join(60) for t in threads]
assert len(seen) == 8 and not any(t.is_alive() for t in threads), seen
assert not any("no address" in s for s in seen), seen
n = len(calls)
call()
assert 1 <= n <= 8 and len(calls) == n and len(seen) == 9
"""
    root = pathlib.Path(__file__).resolve().parents[1]
    subprocess.run([sys.executable, "-W", "ignore", "-c", code], check=True, cwd=root, timeout=240)
