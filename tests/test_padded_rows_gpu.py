"""Projections whose K is not a whole number of packed chunks: the padded copy and the kernels behind it, for every format
that has such shapes, at the ends of a chunk and of the token ranges the kernels divide among themselves."""
import numpy as np
import pytest
import torch

import oracle as o
from gpu_util import dev, run_gemm

pytestmark = pytest.mark.gpu

KS = {o.Q4_0: (32, 224, 288, 2080), o.MLX_4BIT: (32, 288, 2080), o.TERNARY_1_58: (224, 2080), o.MLX_4BIT_G64: (64, 320, 1984),
      o.MLX_4BIT_PLANAR: (96, 2080), o.TERNARY_ROW: (32, 1056), o.PRISM_Q2_0: (128, 1152, 2944)}


def bound(gold):
    """The weights enter as exact sums, the sum is fp32: one fp16 rounding of the result (half an ulp, 2^-11 of it) plus the
    fp32 accumulation of K terms, allowed for as 2^-13 of the largest result."""
    return np.abs(gold) * 2.0 ** -11 + 2.0 ** -13 * np.abs(gold).max() + 2.0 ** -25


@pytest.mark.parametrize("fmt", list(KS))
@pytest.mark.parametrize("M", [1, 2, 128, 129, 300])
def test_padded_rows(bridge, fmt, M):
    for K in KS[fmt]:
        for N in (1, 130, 256):
            X, W = o.baseline_inputs(fmt, M, K, N, 11 + M)
            gold = o.gemm_f64(fmt, X, W, N)
            for _ in range(2):                 # the second call finds the scratch of the first
                Y = run_gemm(bridge, fmt, X, W, N, ex=True).astype(np.float64)
            assert np.all(np.abs(Y - gold) <= bound(gold)), (fmt, M, K, N, np.abs(Y - gold).max())


def test_padded_rows_other_forms(bridge):
    """Head-major output, residual, SwiGLU and packed weights that start on a 2-byte boundary."""
    fmt, M, K, N = o.Q4_0, 70, 544, 192
    X, W = o.baseline_inputs(fmt, M, K, N, 3)
    gold = o.gemm_f64(fmt, X, W, N)
    H = run_gemm(bridge, fmt, X, W, N, layout=1, H=3, D=64).astype(np.float64)
    assert np.all(np.abs(H.transpose(1, 0, 2).reshape(M, N) - gold) <= bound(gold))
    R = np.random.default_rng(4).standard_normal((M, N)).astype(np.float16)
    Y = run_gemm(bridge, fmt, X, W, N, residual=R).astype(np.float64)
    total = gold + R.astype(np.float64)
    assert np.all(np.abs(Y - total) <= bound(total))
    buf = torch.zeros(W.size + 16, dtype=torch.uint8, device="cuda")
    buf[2:2 + W.size] = dev(W)
    Xd, Yd = dev(X), torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    bridge.dispatch_gemm(Xd, buf[2:2 + W.size], Yd, fmt, M, K, N)
    bridge.synchronize()
    assert np.all(np.abs(Yd.cpu().numpy().astype(np.float64) - gold) <= bound(gold))
    _, Wu = o.baseline_inputs(fmt, M, K, N, 5)
    Xs = (X.astype(np.float32) * 0.25).astype(np.float16)
    g, u = o.gemm_f64(fmt, Xs, W, N), o.gemm_f64(fmt, Xs, Wu, N)
    want = g / (1.0 + np.exp(-g)) * u
    Xd, Gd, Ud = dev(Xs), dev(W), dev(Wu)
    bridge.dispatch_swiglu(Xd, Gd, Ud, Yd, fmt, M, K, N)
    bridge.synchronize()
    # the gate's and the up projection's own sums, and the fast exponential and divide of the epilogue (2^-20 relative)
    assert np.all(np.abs(Yd.cpu().numpy().astype(np.float64) - want) <= np.abs(want) * 2.0 ** -10 + 2.0 ** -12 * np.abs(want).max())
    assert bridge.device_error() == 0
