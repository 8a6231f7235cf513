"""The polynomials that take a share of the attention kernel's exponentials, evaluated on the CPU as the kernel does (fp32
multiply-adds, nearest integer through the mantissa), against exp2 in double precision."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
SHIM = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
#include "%s"
template <int DEG> static float ex2(float x) {
    x = std::fmax(x, -120.0f);
    const float r = x + 12582912.0f, n = r - 12582912.0f, f = std::fmaf(n, -1.0f, x);
    float p = exp2poly::coef<DEG>(DEG);
    for (int i = DEG - 1; i >= 0; i--) p = std::fmaf(p, f, exp2poly::coef<DEG>(i));
    uint32_t a, b;
    std::memcpy(&a, &p, 4); std::memcpy(&b, &r, 4);
    a += b << 23;
    std::memcpy(&p, &a, 4);
    return p;
}
extern "C" void ex2_run(int deg, const float* x, float* y, int n) { for (int i = 0; i < n; i++) y[i] = deg == 5 ? ex2<5>(x[i]) : ex2<6>(x[i]); }
"""


# Minimax polynomials, coefficients and multiply-adds rounded to fp32: 7.9e-8 (degree 6, the kernels that follow the running maximum exactly) and
# 1.6e-7 (degree 5); exp2f, in whose place they stand, is documented with two units in the last place (2^-22).
@pytest.mark.parametrize("deg", [6, 5])
def test_exp2_polynomial(tmp_path, deg):
    src, so = tmp_path / "p.cpp", tmp_path / "p.so"
    src.write_text(SHIM % (ROOT / "m4-prefill-engine_b200" / "csrc" / "exp2_poly.cuh"))
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", str(src), "-o", str(so)])
    x = np.concatenate([np.linspace(-3, 0, 3_000_001), np.linspace(-119.99, 8, 1_000_003), [-0.5, 0.5, -1.5, 0.0]]).astype(np.float32)
    y = np.empty_like(x)
    ctypes.CDLL(str(so)).ex2_run(deg, x.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p), len(x))
    want = np.exp2(x.astype(np.float64))
    assert np.abs(y / want - 1).max() <= 2.0 ** -22
    assert y[-1] == 1.0                            # the largest probability of a row stays exactly 1
