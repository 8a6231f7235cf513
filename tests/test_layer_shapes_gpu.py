"""Layers at the ends of their range: one token, hidden sizes that are not whole packed chunks, both head sizes with uneven
numbers of heads, repeated back to back so that one pass's kernels are placed while the other's drain."""
import numpy as np
import pytest

import oracle as o
from gpu_util import dev
from test_layer_gpu import layer_gold_rows, layer_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    dict(M=1, K=512, H=8, Hkv=2, D=64, F=1024), dict(M=1, K=1024, H=8, Hkv=8, D=128, F=768), dict(M=33, K=480, H=6, Hkv=3, D=64, F=1056),
    dict(M=129, K=512, H=6, Hkv=2, D=128, F=544), dict(M=70, K=288, H=5, Hkv=5, D=64, F=320), dict(M=300, K=768, H=3, Hkv=1, D=128, F=1280),
])
def test_layer_shapes(pkg, bridge, case):
    import torch
    from m4_prefill_engine_b200.layer import TransformerLayerConfig, TransformerLayerCoordinator
    M, K, H, Hkv, D, F = (case[k] for k in ("M", "K", "H", "Hkv", "D", "F"))
    w, g = layer_weights(o.Q4_0, K, H, Hkv, D, F)
    rng = np.random.default_rng(3)
    X = (rng.standard_normal((M, K)) * 0.5).astype(np.float16)
    n1, n2 = (rng.uniform(0.5, 1.5, K).astype(np.float16) for _ in range(2))
    layer = TransformerLayerCoordinator(TransformerLayerConfig(M=M, K=K, H=H, D=D, N_mlp=F, attn_scale=D ** -0.5, weight_format=o.Q4_0,
                                                               num_kv_heads=Hkv, rms_eps=1e-5, rope_theta=10000.0, kv_q8_0=True))
    keep = [dev(n1), dev(n2)]
    layer.set_norm_weights(*keep)
    wd, Xd = {k: dev(v) for k, v in w.items()}, dev(X)
    Y = [torch.full((M, K), float("nan"), dtype=torch.float16, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    for y in Y:
        layer.forward(Xd, wd["q"], wd["k"], wd["v"], wd["o"], wd["gate"], wd["up"], wd["down"], y)
    bridge.synchronize()
    assert bridge.device_error() == 0
    assert torch.equal(Y[0], Y[1]) and torch.equal(Y[0], Y[2])
    rows = sorted({0, M // 2, M - 1})
    gold = layer_gold_rows(X, w, n1, n2, rows, H, Hkv, D, F, 1e-5, 10000.0).astype(np.float64)
    diff = np.abs(Y[0].cpu().numpy()[rows].astype(np.float64) - gold)
    # the layer's two residual blocks each round once more than a projection does, and a Q8_0 code on the edge between two
    # integers may fall either way: the pass line of the 8B layer, 2/128 or 2^-7 of the row
    assert np.all(diff <= np.maximum(2.0 / 128, 2.0 ** -7 * np.sqrt(np.mean(gold ** 2, axis=1, keepdims=True))))


@pytest.mark.parametrize("M", [1, 33, 300])
def test_weights_rewritten_just_before(pkg, bridge, M):
    """Packed weights written on the layer's stream right before a forward are the ones it multiplies with, although its projections
    fetch theirs before they wait for the kernel in front."""
    import torch
    from m4_prefill_engine_b200.layer import TransformerLayerConfig, TransformerLayerCoordinator
    K, H, Hkv, D, F = 512, 8, 2, 64, 1024
    sets = [layer_weights(o.Q4_0, K, H, Hkv, D, F)[0]]
    sets.append({k: np.ascontiguousarray(np.roll(v.reshape(-1, 18), 1, axis=0)).reshape(-1) for k, v in sets[0].items()})
    rng = np.random.default_rng(M)
    X = dev((rng.standard_normal((M, K)) * 0.5).astype(np.float16))
    norms = [dev(rng.uniform(0.5, 1.5, K).astype(np.float16)) for _ in range(2)]
    layer = TransformerLayerCoordinator(TransformerLayerConfig(M=M, K=K, H=H, D=D, N_mlp=F, attn_scale=D ** -0.5, weight_format=o.Q4_0,
                                                               num_kv_heads=Hkv, rms_eps=1e-5, rope_theta=10000.0, kv_q8_0=True))
    layer.set_norm_weights(*norms)
    src = [{k: dev(v) for k, v in w.items()} for w in sets]
    names = ("q", "k", "v", "o", "gate", "up", "down")

    def forward(w, y):
        layer.forward(X, *[w[n] for n in names], y)
    want = [torch.empty(M, K, dtype=torch.float16, device="cuda") for _ in range(2)]
    for w, y in zip(src, want):
        forward(w, y)
        bridge.synchronize()
    assert not torch.equal(*want)
    used = {k: v.clone() for k, v in src[0].items()}
    stream = torch.cuda.ExternalStream(bridge.lib.b200_bridge_stream())
    got = [torch.empty(M, K, dtype=torch.float16, device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    for i, y in enumerate(got):
        with torch.cuda.stream(stream):
            for n in names:
                used[n].copy_(src[i & 1][n])
            forward(used, y)
    bridge.synchronize()
    for i, y in enumerate(got):
        assert torch.equal(y, want[i & 1]), i
