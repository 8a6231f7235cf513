"""SwiGLU tiles of the few-token kernel that leave straight from the accumulator: every output row and the ragged ends of features
and tokens, against the same launch on the persistent kernel and the CPU oracle."""
import numpy as np
import pytest

import oracle as o
from gpu_util import check_swiglu
from test_swiglu_attention_gpu import run_swiglu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 16, 17, 127])
@pytest.mark.parametrize("fmt,F", [(o.Q4_0, 9600), (o.TERNARY_ROW, 9506), (o.PRISM_Q2_0, 9473)])
def test_unsplit_tiles(bridge, fmt, F, M):
    K = 1024 if fmt == o.PRISM_Q2_0 else 512                      # more than 148 tiles of 64 features: K is not split
    X, Wg = o.baseline_inputs(fmt, M, K, F, 61)
    _, Wu = o.baseline_inputs(fmt, M, K, F, 62)
    X = (X.astype(np.float32) * 0.25).astype(np.float16)
    g, u = o.gemm_f64(fmt, X, Wg, F), o.gemm_f64(fmt, X, Wu, F)
    scale = max(np.sqrt(np.mean(g ** 2)), np.sqrt(np.mean(u ** 2)), 1.0)
    X = (X.astype(np.float32) / scale).astype(np.float16)       # gate and up of about 1
    out = run_swiglu(bridge, fmt, X, Wg, Wu, F)
    check_swiglu(out, o.gemm_f64(fmt, X, Wg, F), o.gemm_f64(fmt, X, Wu, F), f"unsplit swiglu fmt {fmt} M {M} F {F}")
    bridge.lib.b200_bridge_enable_small_kernel(0)
    try:
        other = run_swiglu(bridge, fmt, X, Wg, Wu, F).astype(np.float64)
    finally:
        bridge.lib.b200_bridge_enable_small_kernel(1)
    # the same fp16 weights, sums of K = 512 or 1024 terms in another order and one rounding to fp16 each
    a, b = out.astype(np.float64), other
    assert np.abs(a - b).max() <= 2.0 ** -10 * max(1.0, np.abs(b).max())
