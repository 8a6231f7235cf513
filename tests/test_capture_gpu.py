"""Launches under stream capture: as the first calls of a process, and replayed after and beside calls that use and grow the
bridge's own scratch."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

PREPARE = r"""
import ctypes, sys
import numpy as np, torch
sys.path.insert(0, %r)
import oracle as o
from __graft_entry__ import load_package
br = load_package().B200Bridge.get_instance()
assert br.init()
L = br.lib
stream = torch.cuda.ExternalStream(L.b200_bridge_stream())
rng = np.random.default_rng(1)
dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
M, F = 20, 128
def proj(K, N):
    X, W = o.baseline_inputs(o.Q4_0, M, K, N, K)
    return dev(X), dev(W), torch.zeros(M, N, dtype=torch.float16, device="cuda"), o.gemm_f64(o.Q4_0, X, W, N)
odd, split = proj(288, 100), proj(1280, 256)
X, Wg = o.baseline_inputs(o.Q4_0, M, 512, F, 7)
X = (X.astype(np.float32) * 0.25).astype(np.float16)
_, Wu = o.baseline_inputs(o.Q4_0, M, 512, F, 8)
sw = dev(X), dev(Wg), dev(Wu), torch.zeros(M, F, dtype=torch.float16, device="cuda")
g, u = o.gemm_f64(o.Q4_0, X, Wg, F), o.gemm_f64(o.Q4_0, X, Wu, F)
att = []
for f16, D, Mq, pos0 in ((True, 128, 1, 2000), (False, 64, 9, 300)):
    Q, K, V = (rng.standard_normal(s, dtype=np.float32).astype(np.float16) for s in ((4, Mq, D), (2, pos0 + Mq, D), (2, pos0 + Mq, D)))
    Kc, Vc = (K, V) if f16 else (o.quantize_q8_0(K), o.quantize_q8_0(V))
    Kx, Vx = (K, V) if f16 else (o.dequantize_q8_0(Kc, K.shape), o.dequantize_q8_0(Vc, V.shape))
    att.append((dev(Q), dev(Kc), dev(Vc), torch.zeros(4, Mq, D, dtype=torch.float16, device="cuda"), Mq, pos0, D, int(f16), o.attention(Q, Kx, Vx, D ** -0.5, pos0, False)))
torch.cuda.synchronize()
def launch_all():
    for x, w, y, _ in (odd, split):
        assert L.m4_bridge_dispatch_gemm(x.data_ptr(), x.numel() * 2, w.data_ptr(), w.numel(), y.data_ptr(), y.numel() * 2, o.Q4_0, M, x.shape[1], y.shape[1]) == 0
    x, a, b, y = sw
    assert L.b200_bridge_dispatch_swiglu(x.data_ptr(), x.numel() * 2, a.data_ptr(), b.data_ptr(), a.numel(), y.data_ptr(), y.numel() * 2, o.Q4_0, M, 512, F) == 0
    for q, k, v, y, Mq, pos0, D, f16, _ in att:
        assert L.b200_bridge_dispatch_attention_q8kv(q.data_ptr(), k.data_ptr(), v.data_ptr(), y.data_ptr(), 4, 2, Mq, pos0 + Mq, D, ctypes.c_float(D ** -0.5), pos0, 0, f16) == 0
outputs = [odd[2], split[2], sw[3]] + [t[3] for t in att]
def verify():
    for x, w, y, gold in (odd, split):
        assert np.abs(y.cpu().numpy() - gold).max() < 2.0 ** -7 * max(1.0, np.abs(gold).max() / 4), "projection"
    assert np.abs(sw[3].cpu().numpy() - g / (1 + np.exp(-g)) * u).max() < 2.0 ** -6 * max(1.0, np.abs(g * u).max() / 8), "swiglu"
    for t in att:
        assert np.abs(t[3].cpu().numpy().astype(np.float64) - t[8].astype(np.float64)).max() < 2.0 ** -9, "attention"
    assert br.device_error() == 0
"""

FIRST = r"""
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=stream):
    launch_all()
graph.replay()
torch.cuda.synchronize()
verify()
"""

LATER = r"""
launch_all()                                     # the bridge's own scratch exists
br.synchronize()
verify()
graphs = [torch.cuda.CUDAGraph() for _ in range(2)]
for graph in graphs:
    with torch.cuda.graph(graph, stream=stream):
        launch_all()
held = L.b200_bridge_graph_scratch_bytes()
assert held > 0
X1, W1 = (dev(t) for t in o.baseline_inputs(o.Q4_0, 300, 2080, 2000, 3))            # a padded copy and a split K, larger than before
Y1 = torch.empty(300, 2000, dtype=torch.float16, device="cuda")
q1 = torch.randn(8, 40, 64, device="cuda").half(); k1 = torch.randn(2, 5040, 64, device="cuda").half(); o1 = torch.empty(8, 40, 64, dtype=torch.float16, device="cuda")
side = torch.cuda.Stream()
torch.cuda.synchronize()
for round in range(20):
    for y in outputs:
        y.fill_(float("nan"))
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graphs[round % 2].replay()               # beside calls on the bridge's stream, which grow and use its scratch
    assert L.m4_bridge_dispatch_gemm(X1.data_ptr(), X1.numel() * 2, W1.data_ptr(), W1.numel(), Y1.data_ptr(), Y1.numel() * 2, o.Q4_0, 300, 2080, 2000) == 0
    assert L.b200_bridge_dispatch_attention_q8kv(q1.data_ptr(), k1.data_ptr(), k1.data_ptr(), o1.data_ptr(), 8, 2, 40, 5040, 64, ctypes.c_float(0.125), 5000, 0, 1) == 0
    torch.cuda.synchronize()
    verify()
    assert bool(torch.isfinite(Y1).all()) and bool(torch.isfinite(o1).all())
assert L.b200_bridge_graph_scratch_bytes() == held
del graph, graphs
import gc, time
gc.collect()
for _ in range(100):                             # (the graphs' resources are given back asynchronously)
    if L.b200_bridge_graph_scratch_bytes() == 0:
        break
    time.sleep(0.05)
assert L.b200_bridge_graph_scratch_bytes() == 0
"""


def run(script):
    r = subprocess.run([sys.executable, "-c", PREPARE % str(ROOT) + script + '\nprint("captured")\n'], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0 and "captured" in r.stdout, r.stdout + r.stderr



def test_first_calls_under_capture():
    """Before anything has been allocated: a K that is not whole chunks, a K of five chunks, SwiGLU of a few tokens, a decode token
    over an fp16 cache, a Q8_0 cache of 64-wide heads."""
    run(FIRST)


def test_replay_beside_and_after_growth():
    """A graph's launches keep scratch of their own: replays beside and after eager calls that use and grow the bridge's, two graphs in
    turn, and the memory given back with the graphs."""
    run(LATER)
