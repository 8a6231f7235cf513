"""The tensor-memory attention kernel at the edges of its query tiles (128 / G positions, two tiles per block), of its key
steps (128) and of the split key range, for both head sizes, against the CPU oracle."""
from ctypes import c_float

import numpy as np
import pytest
import torch

import oracle as o

pytestmark = pytest.mark.gpu
# Outputs are averages of values of about 1: fp16 rounding of O (2^-11) and of P (2^-11 of each term), doubled.
TOL = 2.0 ** -9


@pytest.fixture(scope="module")
def bridge():
    from __graft_entry__ import load_package
    br = load_package().B200Bridge.get_instance()
    assert br.init()
    return br


CASES = [
    # (Hq, Hkv, D, M, pos0, cached tokens behind the last position, fp16 cache, token-major output)
    (4, 4, 64, 1, 0, 0, False, True), (4, 4, 64, 127, 0, 0, False, False), (2, 2, 64, 129, 0, 0, True, True),
    (2, 2, 128, 257, 0, 0, False, True),            # one position past a block of two tiles
    (8, 2, 64, 64, 0, 0, False, True), (8, 2, 64, 65, 63, 0, True, False),
    (6, 2, 64, 85, 43, 0, False, True),             # three heads per kv head: 42 positions and two unused rows per tile
    (10, 2, 128, 51, 0, 0, False, True), (16, 1, 64, 17, 111, 0, False, True), (128, 1, 64, 3, 254, 0, True, True),
    (8, 2, 128, 1, 1535, 0, False, True), (8, 2, 64, 1, 4096, 0, True, False), (24, 8, 128, 2, 2047, 0, False, False),   # split key range
    (4, 2, 64, 130, 1500, 0, False, True), (8, 8, 128, 300, 900, 100, True, True), (8, 2, 128, 70, 3000, 5, False, True),
]


@pytest.mark.parametrize("case", CASES)
def test_attention_edges(bridge, case):
    Hq, Hkv, D, M, pos0, extra, f16, tm = case
    Mkv = pos0 + M + extra
    rng = np.random.default_rng(M * 7 + Mkv)
    Q, K, V = (rng.standard_normal(s, dtype=np.float32).astype(np.float16) for s in ((Hq, M, D), (Hkv, Mkv, D), (Hkv, Mkv, D)))
    scale = D ** -0.5
    if f16:
        Kc, Vc, Kx, Vx = K, V, K, V
    else:
        Kc, Vc = o.quantize_q8_0(K), o.quantize_q8_0(V)
        Kx, Vx = o.dequantize_q8_0(Kc, K.shape), o.dequantize_q8_0(Vc, V.shape)
    gold = o.attention(Q, Kx, Vx, scale, pos0, tm).astype(np.float64)
    Qd, Kd, Vd = (torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (Q, Kc, Vc))
    O = torch.full((M, Hq * D) if tm else (Hq, M, D), float("nan"), dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):                              # the second call reuses the scratch of the first
        assert bridge.lib.b200_bridge_dispatch_attention_q8kv(Qd.data_ptr(), Kd.data_ptr(), Vd.data_ptr(), O.data_ptr(), Hq, Hkv, M, Mkv, D,
                                                              c_float(scale), pos0, int(tm), int(f16)) == 0
    bridge.synchronize()
    assert bridge.device_error() == 0
    got = O.cpu().numpy().astype(np.float64).reshape(gold.shape)
    assert np.all(np.isfinite(got))
    assert np.abs(got - gold).max() <= TOL
