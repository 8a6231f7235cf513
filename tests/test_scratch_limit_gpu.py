"""A GPU without room for scratch (allocations fail through a hook on the host): launches that can do with less take the routes that
need the least, and give the same results."""
import subprocess
import sys
from pathlib import Path

import pytest

from test_capture_gpu import PREPARE

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

CALLS = r"""
L.b200_bridge_debug_limit_scratch.argtypes = [ctypes.c_size_t]
L.b200_bridge_debug_limit_scratch(%d)
launch_all()
br.synchronize()
verify()
"""

LAYER = r"""
sys.path.insert(0, %r)

from test_layer_gpu import layer_weights
from m4_prefill_engine_b200.layer import TransformerLayerConfig, TransformerLayerCoordinator
L.b200_bridge_debug_limit_scratch.argtypes = [ctypes.c_size_t]
for K, H, Hkv, D, F, M in ((480, 6, 3, 64, 1056, 33), (512, 8, 2, 64, 1024, 1024)):
    w, _ = layer_weights(o.Q4_0, K, H, Hkv, D, F)
    wd = {k: dev(v) for k, v in w.items()}
    X = dev((rng.standard_normal((M, K)) * 0.5).astype(np.float16))
    norms = [dev(rng.uniform(0.5, 1.5, K).astype(np.float16)) for _ in range(2)]
    Y = []
    for limit in (0, 1):
        L.b200_bridge_debug_limit_scratch(limit)
        layer = TransformerLayerCoordinator(TransformerLayerConfig(M=M, K=K, H=H, D=D, N_mlp=F, attn_scale=D ** -0.5, weight_format=o.Q4_0,
                                                                   num_kv_heads=Hkv, rms_eps=1e-5, rope_theta=10000.0, kv_q8_0=True))
        layer.set_norm_weights(*norms)
        Y.append(torch.empty(M, K, dtype=torch.float16, device="cuda"))
        torch.cuda.synchronize()
        layer.forward(X, wd["q"], wd["k"], wd["v"], wd["o"], wd["gate"], wd["up"], wd["down"], Y[-1])
        br.synchronize()
    a, b = (y.double() for y in Y)
    # other orders of fp32 sums, fp16 intermediates, and a Q8_0 code on an edge falling either way: the layer's tolerance
    assert float((a - b).norm() / a.norm()) < 3.5e-3, float((a - b).norm() / a.norm())
assert br.device_error() == 0
"""


def run(script):
    r = subprocess.run([sys.executable, "-c", PREPARE % str(ROOT) + script + '\nprint("served")\n'], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0 and "served" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("limit", [1, 400_000])      # nothing; room for the unsplit launch over a Q8_0 cache but not for the rest
def test_calls_without_scratch(limit):
    run(CALLS % limit)


def test_layers_without_scratch():
    run(LAYER % str(ROOT / "tests"))
