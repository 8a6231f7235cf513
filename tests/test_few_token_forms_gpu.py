"""The few-token kernel beyond the single projection: SwiGLU tiles, grouped launches, K splits of unequal length and packed
rings of every depth, against the CPU oracle."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as o
from gpu_util import check, check_swiglu, dev, run_gemm
from test_swiglu_attention_gpu import run_swiglu

pytestmark = pytest.mark.gpu
FORMATS = (o.Q4_0, o.MLX_4BIT, o.Q4_K, o.TERNARY_1_58, o.VAR_RATE_AFFINE, o.EXL3, o.MLX_4BIT_G64, o.MLX_4BIT_PLANAR, o.TERNARY_ROW, o.PRISM_Q2_0)


def rms_factor(fmt):
    return 2.0 if fmt in (o.VAR_RATE_AFFINE, o.EXL3) else 1.0      # weights built from several rounded terms


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("M", [1, 17, 128])
def test_swiglu_few_tokens(bridge, fmt, M):
    unit = 1024 if fmt == o.PRISM_Q2_0 else 256
    for K, F in ((unit, 64), (9 * unit if unit == 256 else 3 * unit, 100), (2 * unit, 1000)):
        X, Wg = o.baseline_inputs(fmt, M, K, F, 21)
        _, Wu = o.baseline_inputs(fmt, M, K, F, 22)
        X = (X.astype(np.float32) * 0.25).astype(np.float16)
        g, u = o.gemm_f64(fmt, X, Wg, F), o.gemm_f64(fmt, X, Wu, F)
        scale = max(np.sqrt(np.mean(g ** 2)), np.sqrt(np.mean(u ** 2)), 1.0)
        X = (X.astype(np.float32) / scale).astype(np.float16)       # gate and up of about 1
        out = run_swiglu(bridge, fmt, X, Wg, Wu, F)
        check_swiglu(out, o.gemm_f64(fmt, X, Wg, F), o.gemm_f64(fmt, X, Wu, F), f"few-token swiglu fmt {fmt} M {M} K {K} F {F}")


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("M", [2, 33, 128])
def test_unequal_splits(bridge, fmt, M):
    unit = 1024 if fmt == o.PRISM_Q2_0 else 256
    for chunks, N in ((3, 130), (7, 64), (13, 300)):
        if unit == 1024 and chunks > 7:
            continue
        X, W = o.baseline_inputs(fmt, M, chunks * unit, N, 31)
        check(run_gemm(bridge, fmt, X, W, N, ex=True), o.gemm_f64(fmt, X, W, N), f"{chunks} chunks fmt {fmt} M {M}", rms_factor=rms_factor(fmt))


@pytest.mark.parametrize("M", [129, 300, 1000])
@pytest.mark.parametrize("small", [0, 1])
def test_unequal_splits_many_tokens(bridge, M, small):
    """Several token tiles: the persistent kernel (shortened token tiles, splits summed by a cluster or by the last CTA) and the
    shapes that go to the few-token kernel instead."""
    bridge.lib.b200_bridge_enable_small_kernel(small)
    try:
        for chunks, N in ((5, 130), (9, 256), (17, 64), (16, 2304), (32, 1100)):
            X, W = o.baseline_inputs(o.Q4_0, M, chunks * 256, N, 33)
            check(run_gemm(bridge, o.Q4_0, X, W, N), o.gemm_f64(o.Q4_0, X, W, N), f"{chunks} chunks M {M} N {N}")
        R = np.random.default_rng(6).standard_normal((M, 1100)).astype(np.float16)
        Y = run_gemm(bridge, o.Q4_0, X, W, N, residual=R)
        check(Y, o.gemm_f64(o.Q4_0, X, W, N) + R.astype(np.float64), f"residual M {M}")
    finally:
        bridge.lib.b200_bridge_enable_small_kernel(1)


@pytest.mark.parametrize("M", [1, 33, 128])
@pytest.mark.parametrize("layout", [0, 1])
def test_grouped_few_tokens(bridge, M, layout):
    vp = ctypes.c_void_p
    for fmt, K, D, Ns in ((o.Q4_0, 1280, 64, (576, 64, 192)), (o.MLX_4BIT, 256, 128, (128, 384)), (o.EXL3, 4096, 128, (512, 128, 128))):
        X, _ = o.baseline_inputs(fmt, M, K, Ns[0], 41)
        Ws = [o.baseline_inputs(fmt, M, K, n, 42 + i)[1] for i, n in enumerate(Ns)]
        Xd, Wd = dev(X), [dev(w) for w in Ws]
        Y = [torch.full((n // D, M, D) if layout else (M, n), float("nan"), dtype=torch.float16, device="cuda") for n in Ns]
        torch.cuda.synchronize()
        c = len(Ns)
        assert bridge.lib.b200_bridge_dispatch_gemm_grouped(Xd.data_ptr(), (vp * c)(*[w.data_ptr() for w in Wd]), (vp * c)(*[y.data_ptr() for y in Y]),
                                                            (ctypes.c_uint32 * c)(*Ns), c, fmt, M, K, layout, D) == 0
        bridge.synchronize()
        assert bridge.device_error() == 0
        for n, w, y in zip(Ns, Ws, Y):
            got = y.cpu().numpy()
            got = got.transpose(1, 0, 2).reshape(M, n) if layout else got
            check(got, o.gemm_f64(fmt, X, w, n), f"grouped fmt {fmt} M {M} N {n}", rms_factor=rms_factor(fmt))


@pytest.mark.parametrize("chunks", [3, 5, 9])
def test_fused_qkv_of_odd_chunk_counts(bridge, chunks):
    """The fused Q/K/V epilogue needs whole sums: a K of an odd number of chunks, which other launches split unequally, stays
    unsplit there and is served."""
    L, M, Hq, Hkv, D, K = bridge.lib, 200, 4, 2, 64, chunks * 256
    X, Wq = o.baseline_inputs(o.Q4_0, M, K, Hq * D, 51)
    Wk, Wv = (o.baseline_inputs(o.Q4_0, M, K, Hkv * D, s)[1] for s in (52, 53))
    Xd, Wd = dev(X), [dev(w) for w in (Wq, Wk, Wv)]
    Q, Kc, Vc = (torch.full((h, M, D), float("nan"), dtype=torch.float16, device="cuda") for h in (Hq, Hkv, Hkv))
    torch.cuda.synchronize()
    assert L.b200_bridge_dispatch_qkv_fused(Xd.data_ptr(), *[w.data_ptr() for w in Wd], Q.data_ptr(), Kc.data_ptr(), Vc.data_ptr(), o.Q4_0, M, K, Hq, Hkv, D,
                                            ctypes.c_float(10000.0), 0, 0, M) == 0
    bridge.synchronize()
    for got, w, h, rope in ((Q, Wq, Hq, True), (Kc, Wk, Hkv, True), (Vc, Wv, Hkv, False)):
        y = o.gemm(o.Q4_0, X, w, h * D, direct_head=True, H=h, D=D)
        y = o.rope(y, 10000.0, 0) if rope else y
        want = y.astype(np.float64)
        # the projection's pass line, once more for the rotation of its rounded values
        assert np.abs(got.cpu().numpy().astype(np.float64) - want).max() <= 2.0 ** -8 * max(1.0, np.sqrt(np.mean(want ** 2)) * 2)
    assert bridge.device_error() == 0
