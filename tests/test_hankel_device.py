"""The device calls that Hankel_long makes beside far_field (the uniform medium's tables, the cumulative
sums) launch with the device of their tensors current.  Without a second GPU: the device contexts are
recorded around a stubbed library call, and the tensors stay on the host."""
import contextlib
import ctypes
import types

import numpy as np
import pytest
import torch

DEV = torch.device("cpu")
MEDIUM = dict(gas="vacuum", absorption_tables="Henke", include_absorption=False, dispersion_tables="Henke",
              include_dispersion=False, n_ir=1.5)


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

    H._uniform_tables_on_device(np.linspace(0, 1e-3, 64), np.linspace(1e16, 2e16, 32), DEV, 1.0, True, **MEDIUM)
    assert recorded == [("mma_hankel_uniform_pre_factor", [DEV])]


def test_uniform_tables_take_one_upload(recorded, monkeypatch):
    """Each pinned copy costs the host some 20 us: the grids and factors of a table go up together."""
    from mma_gb300 import hankel as H

    uploads, args, up = [], [], H._dev
    monkeypatch.setattr(H, "_dev", lambda a, *k: uploads.append(up(a, *k)) or uploads[-1])
    z, w = np.linspace(0, 1e-3, 64), np.linspace(1e16, 2e16, 32)
    monkeypatch.setattr(H, "_sig", lambda: types.SimpleNamespace(mma_hankel_uniform_pre_factor=lambda *a: args.extend(a) or 0))
    H._uniform_tables_on_device(z, w, DEV, 2.0, False, **MEDIUM)
    assert len(uploads) == 1
    at = lambda i, n: np.array((ctypes.c_double * n).from_address(args[i]))  # noqa: E731
    assert args[:2] == [64, 32] and np.array_equal(at(2, 64), z) and np.array_equal(at(3, 32), w)
    assert np.allclose(at(4, 32), 0.5 / H.C_LIGHT) and np.array_equal(at(5, 32), np.zeros(32)) and args[6] == 2.0


@pytest.mark.parametrize("nz, no, cumulative, host", [(2, 768, False, True), (2, 769, False, False),
                                                      (2, 384, True, True), (2, 385, True, False)])
def test_small_uniform_tables_stay_on_the_host(monkeypatch, nz, no, cumulative, host):
    """A call whose tables numpy makes sooner than the device takes pre_factor_table's."""
    from mma_gb300 import hankel as H

    class Stop(Exception):
        pass

    made, got = [], []

    def far_field(*a, **k):
        got.append(a[6])
        raise Stop

    monkeypatch.setattr(H, "_uniform_tables_on_device", lambda *a, **k: made.append(a) or ("device", None))
    monkeypatch.setattr(H, "far_field", far_field)
    z, w = np.linspace(0, 1e-3, nz), np.linspace(1e16, 2e16, no)
    target = types.SimpleNamespace(zgrid=z, ogrid=w, rgrid=np.linspace(0, 1e-4, 8),
                                   source=types.SimpleNamespace(is_cuda=True, device=DEV))
    with pytest.raises(Stop):
        H.Hankel_long(target, 1.0, np.linspace(0, 1e-3, 4), pressure=0.5, store_cumulative_result=cumulative)
    assert len(made) == (0 if host else 1)
    assert np.array_equal(got[0], H.pre_factor_table(z, w, pressure=0.5)[0]) if host else got == ["device"]


@pytest.mark.parametrize("separate", [False, True])
def test_cumulative_sums_run_on_the_planes_device(recorded, separate):
    from mma_gb300 import hankel as H

    P = torch.zeros(4, 5, 3, dtype=torch.complex128)
    planes = [p.clone() for p in P] if separate else list(P)
    H._cumulative(np.linspace(0, 1e-3, 4), planes, np.ones((4, 3)), True)
    assert recorded == [("mma_hankel_cumulative", [DEV])]
