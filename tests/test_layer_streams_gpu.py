"""Two layers of the C++ interface on two streams of their own: neither touches the other's intermediates."""
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include <cuda_runtime.h>
#include "b200_bridge.h"
#include "transformer_layer.h"
using namespace b200_llm;
#define OK(x) do { if (!(x)) { printf("failed: %s\n", #x); return 1; } } while (0)
static void* upload(const std::vector<unsigned char>& h) {
    void* d = nullptr;
    if (cudaMalloc(&d, h.size()) != cudaSuccess || cudaMemcpy(d, h.data(), h.size(), cudaMemcpyHostToDevice) != cudaSuccess) return nullptr;
    return d;
}
static void* q4_0(unsigned n, unsigned k) {          // scales 0x1800 .. 0x1BFF: 2^-9 .. 2^-8
    std::vector<unsigned char> w((size_t)n * (k / 32) * 18);
    for (size_t i = 0; i < w.size(); i++) w[i] = (unsigned char)(rand() >> 7);
    for (size_t i = 0; i < w.size(); i += 18) w[i + 1] = (unsigned char)(0x18 | (w[i + 1] & 3));
    return upload(w);
}
static void* f16(size_t n, int lo, int span) {       // fp16 values with high bytes lo .. lo + span - 1
    std::vector<unsigned char> w(2 * n);
    for (size_t i = 0; i < n; i++) { w[2 * i] = (unsigned char)(rand() >> 7); w[2 * i + 1] = (unsigned char)(lo + (rand() >> 7) % span); }
    return upload(w);
}
int main() {
    OK(m4_bridge_init(nullptr));
    const unsigned M = 2048, K = 512, H = 8, Hkv = 2, D = 64, F = 1024;
    TransformerLayerConfig c;
    c.M = M; c.K = K; c.H = H; c.D = D; c.N_mlp = F; c.num_kv_heads = Hkv; c.rms_eps = 1e-5f; c.rope_theta = 10000.0f; c.kv_q8_0 = true;
    c.attn_scale = 0.125f;
    struct One { cudaStream_t s; TransformerLayerCoordinator* l; void* w[7]; void *x, *y; std::vector<unsigned char> want; } v[2];
    for (One& o : v) {
        OK(cudaStreamCreateWithFlags(&o.s, cudaStreamNonBlocking) == cudaSuccess);
        o.l = new TransformerLayerCoordinator(0, o.s, c);
        OK(o.l->initialize_pipelines());
        const unsigned n[7] = {H * D, Hkv * D, Hkv * D, K, F, F, K}, k[7] = {K, K, K, H * D, K, K, F};
        for (int i = 0; i < 7; i++) OK(o.w[i] = q4_0(n[i], k[i]));
        o.l->set_norm_weights(f16(K, 0x38, 5), f16(K, 0x38, 5));
        OK(o.x = f16((size_t)M * K, 0x34, 8));
        OK(cudaMalloc(&o.y, (size_t)M * K * 2) == cudaSuccess);
        o.want.resize((size_t)M * K * 2);
    }
    auto run = [](One& o) { o.l->forward(o.s, o.x, o.w[0], o.w[1], o.w[2], o.w[3], o.w[4], o.w[5], o.w[6], o.y); return o.l->last_status() == 0; };
    for (One& o : v) {                               // one after the other
        OK(run(o));
        OK(cudaDeviceSynchronize() == cudaSuccess);
        OK(cudaMemcpy(o.want.data(), o.y, o.want.size(), cudaMemcpyDeviceToHost) == cudaSuccess);
    }
    std::vector<unsigned char> got(v[0].want.size());
    for (int round = 0; round < 30; round++) {       // side by side
        for (One& o : v) cudaMemsetAsync(o.y, 0xFF, o.want.size(), o.s);
        for (int i = 0; i < 3; i++) for (One& o : v) OK(run(o));
        OK(cudaDeviceSynchronize() == cudaSuccess);
        for (One& o : v) {
            OK(cudaMemcpy(got.data(), o.y, got.size(), cudaMemcpyDeviceToHost) == cudaSuccess);
            OK(memcmp(got.data(), o.want.data(), got.size()) == 0);
        }
    }
    OK(b200_bridge_device_error() == 0);
    puts("equal");
    return 0;
}
"""


def test_two_layers_on_two_streams(tmp_path, lib_path):
    src, exe = tmp_path / "two.cpp", tmp_path / "two"
    src.write_text(SOURCE)
    cuda = Path("/usr/local/cuda")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "include"), "-I", str(cuda / "include"), str(src), "-o", str(exe),
                           str(lib_path), f"-Wl,-rpath,{Path(lib_path).parent}", "-L", str(cuda / "lib64"), "-lcudart", f"-Wl,-rpath,{cuda / 'lib64'}"])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "equal" in r.stdout, r.stdout + r.stderr
