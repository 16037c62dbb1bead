"""The surrogate's batched calls refuse operands of other types, strides and sizes than
the kernels read, before anything is launched (no GPU: the library is a stand-in)."""
import ctypes
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

BF, F32 = torch.bfloat16, torch.float32


@pytest.fixture
def ops(monkeypatch):
    """sg_ops on CPU tensors, with a library that counts its calls."""
    from mbd_icenav_b200 import sg_ops
    calls = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: calls.append(name) or 0
    monkeypatch.setattr(sg_ops, "lib", lambda: Lib())
    monkeypatch.setattr(sg_ops, "_stream", lambda t: 0)
    monkeypatch.setattr(sg_ops, "_err", lambda d: SimpleNamespace(t=torch.zeros(1, dtype=torch.int32)))
    return SimpleNamespace(conv=sg_ops.conv_forward, dense=sg_ops.dense_forward, grads=sg_ops.weight_grads, calls=calls)


def _dense(**kw):
    z = lambda *s, dtype=BF: torch.zeros(s, dtype=dtype)
    a = dict(x=z(32, 64), w0=z(16, 64), b0=z(16, dtype=F32), out0=z(32, 16), w1=z(8, 16), b1=z(8, dtype=F32),
             out1=z(32, 8, dtype=F32), start=z(4, 16, dtype=F32), row=torch.zeros(32, dtype=torch.int32))
    a.update(kw)
    return a["x"], [(a["w0"], a["b0"], True, a["out0"], a["start"], a["row"]),
                    (a["w1"], a["b1"], False, a["out1"], None, None)]


def test_dense_forward_takes_what_it_reads(ops):
    ops.dense(*_dense())
    ops.dense(*_dense(out1=torch.zeros((32, 8), dtype=BF)))
    ops.dense(*_dense(start=torch.zeros((32, 24)), row=None))
    assert ops.calls == 3 * ["sg_dense_forward"]


@pytest.mark.parametrize("bad", [
    dict(x=torch.zeros((32, 64))), dict(x=torch.zeros((64, 32), dtype=BF).T),
    dict(w0=torch.zeros((16, 64))), dict(w0=torch.zeros((64, 16), dtype=BF).T), dict(w1=torch.zeros((8, 24), dtype=BF)),
    dict(b0=torch.zeros(16, dtype=BF)), dict(b1=torch.zeros(8, dtype=torch.float64)),
    dict(out0=torch.zeros((32, 16))),  # a middle layer's output is the next one's operand
    dict(out0=torch.zeros((16, 32), dtype=BF).T), dict(out1=torch.zeros((32, 8), dtype=torch.float16)),
    dict(out1=torch.zeros((8, 32)).T), dict(out1=torch.zeros((31, 8))),
    dict(start=torch.zeros((4, 16), dtype=BF)), dict(start=torch.zeros((4, 15))), dict(start=torch.zeros((16, 4)).T),
    dict(row=torch.zeros(32, dtype=torch.int64)), dict(row=torch.zeros(64, dtype=torch.int32)[::2]),
    dict(row=torch.zeros(31, dtype=torch.int32)), dict(row=None),
])
def test_dense_forward_refuses(ops, bad):
    with pytest.raises(ValueError):
        ops.dense(*_dense(**bad))
    assert not ops.calls


def _conv(x=None, w=None, b=None, cols=None, act=None):
    z = lambda t, *s, dtype=BF: torch.zeros(s, dtype=dtype) if t is None else t
    return z(x, 2, 8, 8, 1), [(z(w, 8, 64), z(b, 8, dtype=F32), z(cols, 32, 64), z(act, 32, 8))]


def test_conv_forward_takes_what_it_reads(ops):
    ops.conv(*_conv())
    assert ops.calls == ["sg_conv_forward"]


@pytest.mark.parametrize("bad", [
    dict(x=torch.zeros((2, 8, 4, 1), dtype=BF)), dict(x=torch.zeros((2, 8, 16, 1), dtype=BF)),  # not square
    dict(x=torch.zeros((2, 8, 8, 1))), dict(x=torch.zeros((2, 8, 8, 2), dtype=BF)[..., :1]),
    dict(w=torch.zeros((8, 64))), dict(w=torch.zeros((64, 8), dtype=BF).T), dict(b=torch.zeros(8, dtype=BF)),
    dict(cols=torch.zeros((32, 64))), dict(cols=torch.zeros((32, 128), dtype=BF)[:, :64]),
    dict(cols=torch.zeros((16, 64), dtype=BF)), dict(act=torch.zeros((32, 8))),
    dict(act=torch.zeros((32, 16), dtype=BF)[:, :8]),
])
def test_conv_forward_refuses(ops, bad):
    with pytest.raises(ValueError):
        ops.conv(*_conv(**bad))
    assert not ops.calls


@pytest.mark.parametrize("bad", [
    dict(dy=torch.zeros((32, 8))), dict(dy=torch.zeros((8, 32), dtype=BF).T), dict(x=torch.zeros((32, 16))),
    dict(x=torch.zeros((31, 16), dtype=BF)), dict(g=torch.zeros((8, 16), dtype=BF)), dict(g=torch.zeros((16, 8)).T),
    dict(gb=torch.zeros(8, dtype=BF)), dict(gb=torch.zeros(16)[::2]), dict(gb=torch.zeros(7)),
])
def test_weight_grads_refuses(ops, bad):
    a = dict(dy=torch.zeros((32, 8), dtype=BF), x=torch.zeros((32, 16), dtype=BF), g=torch.zeros((8, 16)),
             gb=torch.zeros(8))
    ops.grads([tuple(a.values())])
    assert ops.calls == ["sg_weight_grads"]
    with pytest.raises(ValueError):
        ops.grads([tuple(dict(a, **bad).values())])
    assert len(ops.calls) == 1


def test_a_middle_layer_of_fp32_is_refused_at_the_c_boundary():
    """Before the first layer is launched: its pointers are not looked at."""
    from mbd_icenav_b200 import _abi
    lib = _abi.load_library()
    arr = (_abi.SgDenseLayer * 2)()
    for q in arr:
        q.N, q.K, q.ldw, q.ldd, q.d_dtype = 64, 64, 64, 64, _abi.SG_OUT_F32
        q.w = q.out = 16
    err = ctypes.c_int32()
    assert lib.sg_dense_forward(128, 16, 64, 2, arr, ctypes.addressof(err), None) == _abi.SG_ERR_INVALID
