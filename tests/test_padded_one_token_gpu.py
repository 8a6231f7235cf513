"""One token whose K is not whole chunks: the projection reads the padded copy that the launch in front writes, so two matrices in turn through the
same scratch have to give each its own result, pass after pass."""
import numpy as np
import pytest
import torch

import oracle as o
from gpu_util import check, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,K,N", [(o.Q4_0, 2016, 1024), (o.MLX_4BIT, 1568, 2432), (o.MLX_4BIT, 640, 2919), (o.Q4_0, 960, 2560), (o.TERNARY_1_58, 2080, 4096),
                                     (o.MLX_4BIT_G64, 1088, 2048)])
def test_matrices_in_turn(bridge, fmt, K, N):
    sets = []
    for seed in (1, 2):
        X, W = o.baseline_inputs(fmt, 1, K, N, seed)
        sets.append((dev(X), dev(W), torch.empty(1, N, dtype=torch.float16, device="cuda"), o.gemm_f64(fmt, X, W, N)))
    first = []
    for i in range(60):
        x, w, y, gold = sets[i % 2]
        y.fill_(float("nan"))
        torch.cuda.synchronize()
        bridge.dispatch_gemm_ex(x, w, y, fmt, 1, K, N)
        bridge.synchronize()
        if i < 2:
            first.append(y.clone())
            check(y.cpu().numpy(), gold, f"padded, one token, fmt {fmt} K {K} N {N}", rms_factor=2.0)
        assert torch.equal(y, first[i % 2]), f"pass {i}: {(y != first[i % 2]).sum().item()} of {N} outputs changed"
    assert bridge.device_error() == 0
    assert np.isfinite(first[0].cpu().numpy().astype(np.float32)).all()
