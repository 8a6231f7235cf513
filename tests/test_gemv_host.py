"""Host side of the one-token launches against a CUDA runtime of two devices that runs nothing."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

import oracle as o

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "m4-prefill-engine_b200" / "csrc"


@pytest.fixture(scope="module")
def fake(tmp_path_factory, lib_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    obj = CSRC / "_obj" / "qgemv.o"
    if not Path(nvcc).exists() or not obj.exists():
        pytest.skip("no nvcc, or no objects of the library")
    so = tmp_path_factory.mktemp("fake") / "fake.so"
    inc = Path(nvcc).resolve().parent.parent / "include"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", str(CSRC), "-I", str(ROOT / "include"), "-I", str(inc),
                           str(ROOT / "tests" / "fake_runtime.cpp"), str(obj), "-o", str(so), "-Wl,-Bsymbolic"])
    lib = ctypes.CDLL(str(so))
    lib.fake_smem.restype = ctypes.c_size_t
    return lib


@pytest.mark.parametrize("fmt", [o.MLX_4BIT_G64, o.MLX_4BIT_PLANAR])
def test_second_device_gets_its_shared_memory(fake, fmt):
    """K = 8192 stages more than the 48 KB that a kernel may have without asking: every device has to be asked."""
    for d in (0, 1, 0):
        fake.fake_device(d)
        assert fake.fake_gemv(fmt, 8192, 8192) == 0, f"device {d}"
        assert fake.fake_smem() > 48 * 1024


def test_sm_count_is_asked_once_per_device(fake):
    """The rows per lane follow the SMs of the device that launches, without a query per call."""
    for d in (0, 1):
        fake.fake_device(d)
        assert fake.fake_gemv(o.Q4_0, 512, 512) == 0
    before = fake.fake_queries()
    rows = []
    for d in (0, 1, 0, 1):
        fake.fake_device(d)
        assert fake.fake_gemv(o.Q4_0, 512, 512) == 0
        rows.append(512 // fake.fake_blocks())
    assert rows == [8, 16, 8, 16]                  # 64 warps: fewer than three for each of 148 SMs, more than for each of 2
    assert fake.fake_queries() == before
