"""Infinities, NaN and scales beyond what fp16 holds in projections whose K is not a whole number of packed chunks: the padded
tensor-core launch gives what the CUDA-core kernel gives, which multiplies with fp32 weights."""
import numpy as np
import pytest
import torch

import oracle as o
from gpu_util import dev, run_gemm
from test_swiglu_attention_gpu import run_swiglu

pytestmark = pytest.mark.gpu
FORMATS = (o.Q4_0, o.MLX_4BIT, o.TERNARY_1_58, o.MLX_4BIT_G64, o.MLX_4BIT_PLANAR, o.TERNARY_ROW, o.PRISM_Q2_0)


def both(bridge, call):
    """The default route and the CUDA-core kernel."""
    out = []
    for generic in (0, 1):
        bridge.lib.b200_bridge_force_generic(generic)
        try:
            out.append(call().astype(np.float32))
        finally:
            bridge.lib.b200_bridge_force_generic(0)
    return out


def same(got, want, what):
    for kind, f in (("NaN", np.isnan), ("+inf", np.isposinf), ("-inf", np.isneginf)):
        assert np.array_equal(f(got), f(want)), f"{what}: {kind} {f(got).sum()} against {f(want).sum()}"
    ok = np.isfinite(want)
    # sums of the same fp32 products in another order, one fp16 rounding each
    assert np.all(np.abs(got[ok] - want[ok]) <= np.abs(want[ok]) * 2.0 ** -10 + 2.0 ** -12 * np.abs(want[ok]).max(initial=0.0)), what


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("M", [1, 40, 300])
def test_nonfinite_activations(bridge, fmt, M):
    K, N = (384 if fmt == o.PRISM_Q2_0 else 320), 200
    X, W = o.baseline_inputs(fmt, M, K, N, 5)
    rows = [0] if M == 1 else [1, M // 2, M - 1]
    for i, r in enumerate(rows):
        X[r, (7 * r + 3) % K] = (np.inf, -np.inf, np.nan)[i % 3]
    R = np.random.default_rng(2).standard_normal((M, N)).astype(np.float16)
    got, want = both(bridge, lambda: run_gemm(bridge, fmt, X, W, N, ex=True))
    assert np.isinf(want[rows[0]]).any() or fmt in (o.TERNARY_1_58, o.TERNARY_ROW, o.PRISM_Q2_0)
    same(got, want, "plain")
    same(*both(bridge, lambda: run_gemm(bridge, fmt, X, W, N, residual=R)), "residual")
    same(*both(bridge, lambda: run_gemm(bridge, fmt, X, W, N, layout=1, H=N // 40, D=40)), "heads")
    _, Wu = o.baseline_inputs(fmt, M, K, N, 6)
    Xs = (X.astype(np.float32) * 0.25).astype(np.float16)
    same(*both(bridge, lambda: run_swiglu(bridge, fmt, Xs, W, Wu, N)), "swiglu")


@pytest.mark.parametrize("fmt,size,scale", [(o.Q4_0, 18, 9000.0), (o.MLX_4BIT, 20, 5000.0), (o.Q4_0, 18, np.inf), (o.MLX_4BIT, 20, np.nan)])
@pytest.mark.parametrize("M", [1, 130])
def test_scales_beyond_fp16_products(bridge, fmt, size, scale, M):
    """q * scale overflows fp16, the sum with small activations does not."""
    K, N = 544, 130
    X, W = o.baseline_inputs(fmt, M, K, N, 8)
    X = (X.astype(np.float32) * 2.0 ** -14).astype(np.float16)
    blocks = W.reshape(-1, size)
    blocks[::17, 0:2] = np.frombuffer(np.float16(scale).tobytes(), np.uint8)
    got, want = both(bridge, lambda: run_gemm(bridge, fmt, X, blocks.reshape(-1), N))
    if np.isfinite(scale):
        assert np.isfinite(want).all()
    same(got, want, f"scale {scale}")


def test_residual_in_place(bridge):
    """The residual is the output buffer itself, with an infinite activation in one row."""
    fmt, M, K, N = o.Q4_0, 40, 544, 200
    X, W = o.baseline_inputs(fmt, M, K, N, 4)
    X[7, 9] = np.inf
    R = np.random.default_rng(3).standard_normal((M, N)).astype(np.float16)

    def call():
        Xd, Wd, Y = dev(X), dev(W), dev(R)
        torch.cuda.synchronize()
        bridge.dispatch_gemm_ex(Xd, Wd, Y, fmt, M, K, N, 0, 0, 0, Y)
        bridge.synchronize()
        return Y.cpu().numpy()
    same(*both(bridge, call), "in place")
