"""Tensors in host memory are refused where a launch takes its stream (no GPU needed)."""
import pytest

torch = pytest.importorskip("torch")


def test_current_stream_refuses_the_cpu():
    from mbd_icenav_b200 import _abi
    with pytest.raises(ValueError, match="cuda device"):
        _abi.current_stream(torch.device("cpu"))


def test_launches_on_host_tensors_are_refused(monkeypatch):
    """Through the calls themselves, with a library that would take any pointer."""
    from types import SimpleNamespace
    from mbd_icenav_b200 import rollouts, sg_ops
    called = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: called.append(name) or 0
    monkeypatch.setattr(sg_ops, "lib", lambda: Lib())
    monkeypatch.setattr(rollouts._abi, "load_library", lambda: Lib())
    monkeypatch.setattr(rollouts, "_device_grid", lambda c: c.grid)
    # as on a machine with a GPU, where the current device's stream can always be had
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda i: 0, raising=False)
    bf = lambda *s: torch.zeros(s, dtype=torch.bfloat16)
    cm = SimpleNamespace(grid=torch.zeros(4, 4), x_origin=0.0, y_origin=0.0, resolution=1.0, rows=4, cols=4)
    for call in (lambda: sg_ops.gemm(bf(8, 64), bf(8, 64)), lambda: sg_ops.transpose(bf(8, 8)),
                 lambda: sg_ops.pack_rows(None, torch.zeros(4, 3), bf(4, 8)),
                 lambda: rollouts.waypoint_costs(torch.zeros(3, 2, 3), cm)):
        with pytest.raises(ValueError, match="cuda device"):
            call()
    assert not called
