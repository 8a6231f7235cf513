"""A projection whose activation rows never arrive (flags that nothing sets, the wait limited to 50 ms): the persistent kernel returns with
code 110, writes no row that was waited for, raises no arrival flag, and the next launch is served.  Ranks are buffers on one GPU; nothing
waits on another launch."""
import ctypes
import time

import numpy as np
import pytest
import torch

import oracle as o
from gpu_util import check, check_swiglu, dev

pytestmark = pytest.mark.gpu


def _arr(xs):
    return (ctypes.c_void_p * len(xs))(*[int(x) for x in xs])


# late: owners whose rows never come; rows of an owner are M / world.  World 8: 128 rows, so that of a CTA pair's 256 tokens the odd CTA's alone are late.
@pytest.mark.parametrize("kind,fmt,M,K,N,world,late,pair", [
    ("plain", o.Q4_0, 1024, 1024, 8192, 8, (7,), 1),
    ("plain", o.Q4_0, 1024, 1024, 8192, 8, (0, 2, 4, 6), 1),
    ("plain", o.Q4_0, 1024, 1024, 8192, 8, (1, 3, 5, 7), 1),
    ("plain", o.VAR_RATE_AFFINE, 1024, 512, 8192, 2, (1,), 1),
    ("plain", o.Q4_0, 1024, 1024, 8192, 2, (0, 1), 0),
    ("plain", o.TERNARY_ROW, 1000, 512, 9600, 2, (1,), 0),
    ("swiglu", o.Q4_0, 1024, 1024, 4096, 2, (1,), 1),
    ("swiglu", o.Q4_K, 1024, 1024, 4096, 8, (3, 7), 0),
    ("scatter", o.Q4_0, 1024, 1024, 8192, 2, (0, 1), 1),
    ("scatter", o.Q4_0, 1024, 1024, 1024, 2, (0, 1), 0),
])
def test_late_rows(bridge, pkg, kind, fmt, M, K, N, world, late, pair):
    from m4_prefill_engine_b200.layer import _bind_layer
    L = bridge.lib
    _bind_layer(L)
    L.b200_peer_set_wait_limit_ms.argtypes = [ctypes.c_uint]
    L.b200_peer_set_wait_limit_ms.restype = None
    X, W = o.baseline_inputs(fmt, M, K, N, 17)
    X = (X.astype(np.float32) * 0.25).astype(np.float16)
    Wu = o.baseline_inputs(fmt, 1, K, N, 18)[1] if kind == "swiglu" else None
    Xd, Wd, Wud = dev(X), dev(W), dev(Wu) if Wu is not None else None
    rows, epoch = M // world, 5
    Y = torch.full((M, N), 3.0, dtype=torch.float16, device="cuda")
    flags = [torch.zeros(16, dtype=torch.int32, device="cuda") for _ in range(world)]
    flags[0][8:8 + world] = epoch
    for r in late:
        flags[0][8 + r] = epoch - 1
    recv = [torch.full((world, rows, N), 3.0, dtype=torch.float32, device="cuda") for _ in range(world)] if kind == "scatter" else None
    torch.cuda.synchronize()

    def launch():
        return L.b200_peer_gemm_wait_rows(Xd.data_ptr(), Wd.data_ptr(), Wud.data_ptr() if Wud is not None else None, Y.data_ptr(), fmt, M, K, N, 0, world,
                                          _arr([t.data_ptr() for t in recv]) if recv else None, _arr([f.data_ptr() for f in flags]), epoch)

    assert bridge.device_error() == 0
    L.b200_bridge_enable_pair_kernel(pair)
    L.b200_peer_set_wait_limit_ms(50)
    try:
        t0 = time.perf_counter()
        assert launch() == 0
        assert (L.b200_bridge_last_launch_pair() > 0) == bool(pair)
        bridge.synchronize()
        assert time.perf_counter() - t0 < 6.0                       # the other CTA of a pair gives up after its own second
        assert bridge.device_error() == 110
        part = Y.cpu().numpy()
        if kind == "scatter":
            assert all(float(t.min()) == 3.0 and float(t.max()) == 3.0 for t in recv)
            assert all(f[:8].cpu().tolist() == [0] * 8 for f in flags)
        for r in late:
            assert (part[r * rows:(r + 1) * rows] == 3.0).all(), f"rows of owner {r} were written"
        assert L.b200_bridge_clear_device_error() == 0
        # the rows are there now: the same launch is served
        flags[0][8:8 + world] = epoch
        torch.cuda.synchronize()
        assert launch() == 0
        bridge.synchronize()
        assert bridge.device_error() == 0
    finally:
        L.b200_peer_set_wait_limit_ms(0)
        L.b200_bridge_enable_pair_kernel(1)
        L.b200_bridge_clear_device_error()
    full = Y.cpu().numpy()
    if kind == "scatter":
        assert all(f[:8].cpu().tolist() == [epoch] + [0] * 7 for f in flags)
        full = np.concatenate([t[0].cpu().numpy() for t in recv]).astype(np.float16)
    if kind == "swiglu":
        check_swiglu(full, o.gemm_f64(fmt, X, W, N), o.gemm_f64(fmt, X, Wu, N), f"late rows swiglu fmt {fmt}")
    else:
        check(full, o.gemm_f64(fmt, X, W, N), f"late rows {kind} fmt {fmt}", rms_factor=2.0 if fmt == o.VAR_RATE_AFFINE else 1.0)
        if kind == "plain":                                           # what the aborted launch did write are whole tiles
            assert ((part == full) | (part == 3.0)).all()
