"""The tensor-memory attention kernel at the edges of its query tiles (128 / G positions, two tiles per block), of its key
steps (128) and of the split key range, for both head sizes, against the CPU oracle."""
from ctypes import c_float, c_size_t

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
    (8, 2, 64, 3, 700, 5000, False, True), (6, 3, 128, 200, 0, 777, False, False),                                      # a long tail that no row sees
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


def test_unseen_cache_is_not_expanded(bridge):
    """A cache laid out for 60000 tokens, 4008 of them in use: the call needs scratch for those only."""
    L, Hq, Hkv, D, M, pos0, Mkv = bridge.lib, 8, 2, 128, 8, 4000, 60000
    rng = np.random.default_rng(5)
    Q = rng.standard_normal((Hq, M, D), dtype=np.float32).astype(np.float16)
    K, V = (rng.standard_normal((Hkv, pos0 + M, D), dtype=np.float32).astype(np.float16) for _ in range(2))
    used = [o.quantize_q8_0(t).reshape(Hkv, -1) for t in (K, V)]
    cache = [torch.full((Hkv, Mkv * D // 32 * 34), 0xFF, dtype=torch.uint8, device="cuda") for _ in used]       # NaN scales behind what is in use
    for c, u in zip(cache, used):
        c[:, :u.shape[1]] = torch.from_numpy(u).cuda()
    gold = o.attention(Q, *(o.dequantize_q8_0(u.reshape(-1), K.shape) for u in used), D ** -0.5, pos0, False).astype(np.float64)
    Qd, O = torch.from_numpy(Q).cuda(), torch.empty(Hq, M, D, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    L.b200_bridge_debug_limit_scratch.argtypes = [c_size_t]
    L.b200_bridge_debug_limit_scratch(32 << 20)              # the whole cache would take 61 MB
    try:
        assert L.b200_bridge_dispatch_attention_q8kv(Qd.data_ptr(), cache[0].data_ptr(), cache[1].data_ptr(), O.data_ptr(), Hq, Hkv, M, Mkv, D,
                                                     c_float(D ** -0.5), pos0, 0, 0) == 0
        launches = L.b200_bridge_attention_launches()
    finally:
        L.b200_bridge_debug_limit_scratch(0)
    bridge.synchronize()
    assert launches == 3                                     # expansion, split attention, combination: not the kernels without scratch
    assert np.abs(O.cpu().numpy().astype(np.float64) - gold).max() <= TOL


@pytest.mark.parametrize("Hq,Hkv,D,M,pos0", [(4, 2, 64, 200, 0), (6, 2, 64, 90, 300), (3, 1, 128, 150, 100), (8, 2, 128, 200, 0), (4, 4, 128, 3, 1500)])
@pytest.mark.parametrize("where", ["q", 0, 3])          # 0, 3: a key whose exponential comes from the special-function unit, from the polynomial
def test_nonfinite_scores(bridge, Hq, Hkv, D, M, pos0, where):
    """NaN and infinities in Q or K: the rows that the warp-level kernels answer with NaN, and no others."""
    L, Mkv = bridge.lib, pos0 + M
    rng = np.random.default_rng(M)
    Q, K, V = (rng.standard_normal(s, dtype=np.float32).astype(np.float16) for s in ((Hq, M, D), (Hkv, Mkv, D), (Hkv, Mkv, D)))
    if where == "q":
        Q[1, M // 2, 5], Q[0, M - 1, 0] = np.nan, np.inf
    else:
        K[0, pos0 // 8 * 8 + where, 7] = np.nan
        K[Hkv - 1, Mkv - 2, 3] = -np.inf
    Qd, Kd, Vd = (torch.from_numpy(t).cuda() for t in (Q, K, V))
    out = []
    for hook in (0, 1):
        O = torch.empty(Hq, M, D, dtype=torch.float16, device="cuda")
        torch.cuda.synchronize()
        L.b200_bridge_force_legacy_attention(hook)
        try:
            assert L.b200_bridge_dispatch_attention_q8kv(Qd.data_ptr(), Kd.data_ptr(), Vd.data_ptr(), O.data_ptr(), Hq, Hkv, M, Mkv, D, c_float(D ** -0.5), pos0, 0, 1) == 0
        finally:
            L.b200_bridge_force_legacy_attention(0)
        bridge.synchronize()
        out.append(O.cpu().numpy().astype(np.float64))
    assert np.isnan(out[1]).any()
    assert np.array_equal(np.isnan(out[0]), np.isnan(out[1]))
    ok = ~np.isnan(out[1])
    assert np.all(np.isfinite(out[0][ok])) and np.abs(out[0][ok] - out[1][ok]).max(initial=0.0) <= TOL
