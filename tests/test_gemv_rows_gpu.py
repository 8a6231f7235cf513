"""One token: rows per lane and the staged copies of 128-byte chunks, at the sizes where the choice turns and the last rows and chunks are ragged,
against the CPU oracle."""
import numpy as np
import pytest

import oracle as o
from gpu_util import check, run_gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [o.Q4_0, o.Q4_K, o.TERNARY_1_58, o.MLX_4BIT_G64, o.TERNARY_ROW, o.MLX_4BIT_PLANAR])
@pytest.mark.parametrize("K,N", [(256, 1), (512, 3551), (512, 3553), (768, 4736), (768, 4745), (1280, 1775), (1280, 2377), (8192, 441), (8192, 599), (8448, 57)])
def test_one_token(bridge, fmt, K, N):
    X, W = o.baseline_inputs(fmt, 1, K, N, 71)
    check(run_gemm(bridge, fmt, X, W, N, ex=True), o.gemm_f64(fmt, X, W, N), f"one token, fmt {fmt} K {K} N {N}")
