"""M4QuantizedLinear when a kernel reports that it gave up: zeros where nothing was written, never memory as it was found (on the
CPU, with the library replaced by a stand-in)."""
from ctypes import c_int

import pytest
import torch

import oracle as o


class Bridge:
    """Stands in for the library: the projection of call `failing` writes nothing and reports code 106."""

    def __init__(self, failing):
        self.calls, self.failing, self.error_seen = 0, failing, c_int(0)

    def is_initialized(self):
        return True

    def dispatch(self, x, w, y, *args, **kwargs):
        if self.calls == self.failing:
            self.error_seen.value = 106
        else:
            y.fill_(3.0)
        self.calls += 1
        return 0


@pytest.mark.parametrize("shape", [(64,), (1, 64), (2, 3, 64)])
def test_no_unwritten_memory(pkg, monkeypatch, shape):
    from m4_prefill_engine_b200 import modules
    b = Bridge(failing=1)
    monkeypatch.setattr(modules.B200Bridge, "get_instance", classmethod(lambda cls: b))
    monkeypatch.setattr(modules, "m4_bridge_dispatch_gemm", b.dispatch)
    monkeypatch.setattr(modules, "m4_bridge_dispatch_gemv", b.dispatch)
    monkeypatch.setattr(modules, "m4_bridge_synchronize", lambda: None)
    empty = torch.empty
    monkeypatch.setattr(modules.torch, "empty", lambda *a, **k: empty(*a, **k).fill_(float("nan")))
    lin = modules.M4QuantizedLinear(64, 32, format=o.Q4_0, device="cpu")
    x = torch.ones(shape)
    assert torch.equal(lin(x), torch.full((*shape[:-1], 32), 3.0, dtype=torch.float16))
    assert torch.equal(lin(x), torch.zeros((*shape[:-1], 32), dtype=torch.float16))      # the call that failed
    assert torch.equal(lin(x), torch.full((*shape[:-1], 32), 3.0, dtype=torch.float16))  # a good one behind it
    assert torch.equal(lin(x, check_finite=True), torch.full((*shape[:-1], 32), 3.0, dtype=torch.float16))
