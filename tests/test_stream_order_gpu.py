"""The bridge's work is ordered behind the caller's stream on the GPU, without a wait on the host."""
import pytest
import torch

import oracle as o
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [False, True])
def test_inputs_still_being_produced(bridge, side):
    """X is overwritten by torch work that is still queued (tens of milliseconds of it) when the projection is dispatched, on the
    default stream and on a side stream; the projection reads what that work leaves."""
    M, K, N = 40, 512, 256
    X, W = o.baseline_inputs(o.Q4_0, M, K, N, 5)
    Xf, Wd = dev(X), dev(W)
    want = torch.empty(M, N, dtype=torch.float16, device="cuda")
    bridge.dispatch_gemm(Xf, Wd, want, o.Q4_0)
    bridge.synchronize()
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        a = torch.tanh(torch.randn(4096, 4096, device="cuda"))
        a = torch.tanh(a @ a)                       # libraries and modules are loaded before the queue is filled
        (Xf + (a.sum() * 0).to(torch.float16)).clone()
        x = torch.zeros_like(Xf)
        got = torch.empty_like(want)
        torch.cuda.synchronize()
        for _ in range(60):
            a = torch.tanh(a @ a)
        x.copy_(Xf + (a.sum() * 0).to(torch.float16))
        busy = not stream.query()
        bridge.dispatch_gemm(x, Wd, got, o.Q4_0)
        still = not stream.query()
        bridge.synchronize()
    assert busy and still, "the dispatch waited on the host"
    assert torch.equal(got, want)


def test_stream_under_capture_is_refused(bridge):
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    t = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        rc = bridge.lib.b200_bridge_wait_stream(torch.cuda.current_stream().cuda_stream)
        t.add_(1)
    assert rc == -6
    g.replay()
    torch.cuda.synchronize()
    assert float(t.sum()) == 8.0


def test_bridge_stream_under_capture_is_left_alone(bridge):
    """The bridge's own stream is being captured and the caller's stream is busy: no edge from uncaptured work may enter the capture."""
    own = torch.cuda.ExternalStream(bridge.lib.b200_bridge_stream())
    side, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    t = torch.zeros(8, device="cuda")
    with torch.cuda.stream(own):
        t.add_(0)                                   # the kernel is loaded before the capture
    with torch.cuda.stream(side):
        torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=own):
        with torch.cuda.stream(side):
            torch.cuda._sleep(200_000_000)          # about a tenth of a second
        rc = bridge.lib.b200_bridge_wait_stream(side.cuda_stream)
        t.add_(1)
    assert rc == -6
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert float(t.sum()) == 8.0


def test_other_captures_are_left_alone(bridge):
    """A capture on a stream that the bridge has nothing to do with goes on while the bridge waits for idle and busy streams."""
    own, busy, idle, g = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    t = torch.zeros(8, device="cuda")
    with torch.cuda.stream(own):
        t.add_(0)
    with torch.cuda.stream(busy):
        torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=own):
        with torch.cuda.stream(busy):
            torch.cuda._sleep(200_000_000)
        rc = [bridge.lib.b200_bridge_wait_stream(s.cuda_stream) for s in (idle, busy)]
        t.add_(1)
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert rc == [0, 0] and float(t.sum()) == 8.0


def test_module_under_capture_takes_the_calls_one_by_one(bridge):
    """M4QuantizedLinear.forward in one call of the library: behind a busy torch stream, and refused (nothing enqueued) for a captured one."""
    from m4_prefill_engine_b200.modules import M4QuantizedLinear
    import oracle as o
    X, W = o.baseline_inputs(o.Q4_0, 1, 512, 256, 5)
    lin = M4QuantizedLinear(512, 256, format=o.Q4_0, weight=torch.from_numpy(W.reshape(-1).view("uint8").copy()))
    want = lin(torch.from_numpy(X).cuda()).clone()
    x, s, g, t = torch.zeros(1, 512, dtype=torch.float16, device="cuda"), torch.cuda.Stream(), torch.cuda.CUDAGraph(), torch.zeros(8, device="cuda")
    src = torch.from_numpy(X).cuda()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)               # about ten milliseconds: the input is written behind it
        x.copy_(src)
        got = lin(x)
    assert torch.equal(got, want)
    y = torch.zeros(1, 256, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=torch.cuda.Stream()):
        served = bridge.project(x, lin.weight, y, 0, 1, 512, 256)
        t.add_(1)
    g.replay()
    torch.cuda.synchronize()
    assert served is False and float(y.abs().max()) == 0.0 and float(t.sum()) == 8.0
