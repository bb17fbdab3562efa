"""Order of torch's stream and the library's where arrays on the device change
hands, on the CPU: a fake library that refuses arrays whose conversion nobody
waited for."""
import types

import numpy as np
import pytest
import torch

from openswpc_b200 import adjoint
from tests.models import small3d


@pytest.mark.parametrize("form", ["float32", "float64", "transposed"])
def test_library_reads_converted_models_after_a_wait(form, monkeypatch):
    """Every model array handed to the library was there before the call or
    was converted and waited for; so was the memory of the gradients."""
    p = small3d(nx=20, ny=18, nz=12, na=4, nt=4)
    shape = (p.ny + 6, p.nx + 6, p.nz + 6)
    prob = adjoint.Misfit3D.__new__(adjoint.Misfit3D)
    pending, calls = set(), []
    to_dev, empty = adjoint.Misfit3D._dev, torch.empty

    def dev(self, a):
        t = to_dev(self, a)
        if not isinstance(a, torch.Tensor) or t.data_ptr() != a.data_ptr():
            pending.add(t.data_ptr())
        return t

    def new(*a, **k):
        t = empty(*a, **k)
        pending.add(t.data_ptr())   # torch may still be using that memory
        return t

    class Lib:
        def __getattr__(self, name):
            def call(*args):
                for a in args:
                    assert getattr(a, "value", None) not in pending or a.value is None, name
                calls.append(name)
                return 0
            return call

    monkeypatch.setattr(adjoint.Misfit3D, "_dev", dev)
    monkeypatch.setattr(adjoint.Misfit3D, "_on_device", lambda self, *ts: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: types.SimpleNamespace(synchronize=pending.clear))
    monkeypatch.setattr(torch, "empty", new)
    prob.p, prob.ckpt, prob.device = p, 4, "cpu"
    prob.qp = prob.qs = np.ones(shape, np.float32)
    prob.obs = np.zeros((1, 3, 1), np.float32)
    prob.solver = types.SimpleNamespace(ctx=None, lib=Lib(), medium=None)
    model = [torch.ones(shape, dtype=torch.float64 if form == "float64" else torch.float32) for _ in range(3)]
    if form == "transposed":
        model = [torch.ones(shape[::-1]).permute(2, 1, 0) for _ in range(3)]
    prob.gradient(*model)
    assert calls[0] == "swpc_vmodel_velocity_device" and calls[-1] == "swpc_gradient_model_device"


def test_library_reads_the_perturbation_after_a_wait(monkeypatch):
    """A CUDA perturbation xi, which torch may still be writing on its stream,
    is waited for before the medium set-up reads it."""
    from openswpc_b200.swpc3d import DeviceMedium
    p = small3d(nx=20, ny=18, nz=12, na=4, nt=4)
    waited, calls = [], []

    class Lib:
        def __getattr__(self, name):
            def call(*args):
                assert waited, name
                calls.append(name)
                return 0
            return call

    xi = types.SimpleNamespace(shape=(p.ny + 6, p.nx + 6, p.nz + 6), dtype=torch.float32, is_cuda=True, device="cuda:0",
                               data_ptr=lambda: 256, is_contiguous=lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream",
                        lambda d=None: types.SimpleNamespace(synchronize=lambda: waited.append(d)))
    DeviceMedium(Lib(), None, p, xi)
    assert calls[0] == "swpc_vmodel_lhm_device_opt" and waited == ["cuda:0"]
