"""The device calls that Hankel_long makes beside far_field (the uniform medium's tables, the cumulative
sums) launch with the device of their tensors current.  Without a second GPU: the device contexts are
recorded around a stubbed library call, and the tensors stay on the host."""
import contextlib
import types

import numpy as np
import pytest
import torch

DEV = torch.device("cpu")


@pytest.fixture
def recorded(monkeypatch):
    """(current, calls): the stack of devices made current, and per library call its state then."""
    from mma_gb300 import hankel as H

    current, calls = [], []

    @contextlib.contextmanager
    def device(dev):
        current.append(dev)
        yield
        current.pop()

    class Lib:
        def __getattr__(self, name):
            return lambda *a: calls.append((name, list(current))) or 0

    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: types.SimpleNamespace(cuda_stream=0))
    monkeypatch.setattr(H, "_sig", Lib)
    monkeypatch.setattr(H, "_dev", lambda a, dev, dtype=torch.float64: torch.as_tensor(np.array(a), dtype=dtype))
    return calls


def test_uniform_tables_run_on_the_source_device(recorded):
    from mma_gb300 import hankel as H

    H._uniform_tables_on_device(np.linspace(0, 1e-3, 4), np.linspace(1e16, 2e16, 3), DEV, 1.0, True, gas="vacuum",
                                absorption_tables="Henke", include_absorption=False, dispersion_tables="Henke",
                                include_dispersion=False, n_ir=1.0)
    assert recorded == [("mma_hankel_uniform_pre_factor", [DEV])]


@pytest.mark.parametrize("separate", [False, True])
def test_cumulative_sums_run_on_the_planes_device(recorded, separate):
    from mma_gb300 import hankel as H

    P = torch.zeros(4, 5, 3, dtype=torch.complex128)
    planes = [p.clone() for p in P] if separate else list(P)
    H._cumulative(np.linspace(0, 1e-3, 4), planes, np.ones((4, 3)), True)
    assert recorded == [("mma_hankel_cumulative", [DEV])]
