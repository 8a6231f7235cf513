// C ABI of the bridge (include/b200_bridge.h): argument validation in the reference's order
// (core/bridge/m4_mlx_bridge.mm:194-230), host/device pointer resolution, staging, and dispatch
// onto the kernels.  One compute stream plus two copy streams for host buffers; a mutex guards all state, as in the reference
// (core/bridge/m4_mlx_bridge.mm:20,84,284-287).
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstring>
#include <list>
#include <mutex>
#include <string>
#include <unordered_map>

#include "../../include/b200_bridge.h"
#include "../../include/quant_router.h"
#include "bridge_state.cuh"
#include "layer_ops.cuh"
#include "qgemm.cuh"

namespace bridge {

State g;

cudaError_t scratch_malloc(void** p, size_t bytes) {
    const size_t limit = g.scratch_limit;
    if (limit && bytes > limit) { *p = nullptr; return cudaErrorMemoryAllocation; }
    const cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) { cudaGetLastError(); *p = nullptr; }
    return e;
}

bool DevBuf::ensure(size_t n) {
    if (n <= cap) return true;
    if (p) cudaFree(p);        // implicit device sync: nothing in flight still uses the old block
    p = nullptr; cap = 0;
    size_t want = n + n / 4;
    if (scratch_malloc(&p, want) != cudaSuccess) return false;
    cap = want;
    return true;
}
void DevBuf::release() { if (p) cudaFree(p); p = nullptr; cap = 0; }

void set_error(const std::string& s) { g.last_error = s; }

bool is_device_ptr(const void* ptr) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, ptr) != cudaSuccess) { cudaGetLastError(); return false; }
    return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
}

// Device address for an input buffer: the pointer itself when it is device memory, the
// registered device copy when it is a registered host weight buffer, else a staged copy.
const void* resolve_in(const void* ptr, size_t bytes, DevBuf& stage, bool weights, int* rc) {
    if (is_device_ptr(ptr)) return ptr;
    if (weights) {
        auto it = g.registered.find(ptr);
        if (it != g.registered.end() && it->second.bytes >= bytes) return it->second.dev;
    }
    // a projection's copy back may still be writing the host buffer this call reads
    for (StageSlot& sl : g.slots)
        if (sl.out_pending) cudaStreamWaitEvent(g.stream, sl.ev_out, 0);
    if (!stage.ensure(bytes)) { *rc = -5; return nullptr; }
    if (cudaMemcpyAsync(stage.p, ptr, bytes, cudaMemcpyHostToDevice, g.stream) != cudaSuccess) {
        cudaGetLastError(); *rc = -5; return nullptr;
    }
    g.h2d_bytes += bytes;
    return stage.p;
}

// Device address to write an output into; `*host_dst` is set when a copy back is needed.
void* resolve_out(void* ptr, size_t bytes, DevBuf& stage, void** host_dst, int* rc) {
    *host_dst = nullptr;
    if (is_device_ptr(ptr)) return ptr;
    if (!stage.ensure(bytes)) { *rc = -5; return nullptr; }
    *host_dst = ptr;
    return stage.p;
}

int copy_back(void* host_dst, const void* dev_src, size_t bytes) {
    if (cudaMemcpyAsync(host_dst, dev_src, bytes, cudaMemcpyDeviceToHost, g.stream) != cudaSuccess) { cudaGetLastError(); return -5; }
    g.d2h_bytes += bytes;
    cudaEventRecord(g.ev_main_d2h, g.stream);
    g.main_d2h_pending = true;
    g.main_d2h_seq = ++g.dispatch_seq;
    return 0;
}

namespace {

inline bool overlaps(const void* a, size_t an, const char* b, size_t bn) {
    const char* ac = static_cast<const char*>(a);
    return b && ac < b + bn && b < ac + an;
}

// Host input of a pipelined projection call: staged on the copy-in stream into the slot's buffer.
const void* stage_in(const void* ptr, size_t bytes, StageSlot& sl, DevBuf& buf, bool weights, bool* staged, int* rc) {
    if (is_device_ptr(ptr)) return ptr;
    if (weights) {
        auto it = g.registered.find(ptr);
        if (it != g.registered.end() && it->second.bytes >= bytes) return it->second.dev;
    }
    // ordering through host memory: an earlier call's result may still be on its way into this buffer
    for (StageSlot& o : g.slots)
        if (o.out_pending && overlaps(ptr, bytes, o.out_ptr, o.out_bytes)) cudaStreamWaitEvent(g.stream_in, o.ev_out, 0);
    if (!*staged) {     // first upload of this call: the slot's buffers must be free, earlier host results complete
        if (sl.used) cudaStreamWaitEvent(g.stream_in, sl.ev_kernel, 0);
        if (g.main_d2h_pending) cudaStreamWaitEvent(g.stream_in, g.ev_main_d2h, 0);
    }
    if (!buf.ensure(bytes)) { *rc = -5; return nullptr; }
    g.copies = true; g.copy_seq++;
    if (cudaMemcpyAsync(buf.p, ptr, bytes, cudaMemcpyHostToDevice, g.stream_in) != cudaSuccess) { cudaGetLastError(); *rc = -5; return nullptr; }
    g.h2d_bytes += bytes;
    *staged = true;
    return buf.p;
}

}  // namespace

bool capturing(cudaStream_t stream) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) { cudaGetLastError(); return false; }
    return cap != cudaStreamCaptureStatusNone;
}

namespace {

// Blocks of captured graphs.  A graph holds its block through a user object, whose destructor may not call into CUDA: it marks the
// block, and the next launch outside a capture frees it (or the next capture takes it over).
struct GraphBlock { unsigned long long capture; uint8_t* p; size_t bytes; std::atomic<bool> released; };
std::list<GraphBlock> graph_blocks;                         // (under State::mu; entries do not move)
constexpr size_t COUNTER_BYTES = 4096 * sizeof(uint32_t);    // in front of a block's scratch

// cudaMalloc and cudaFree are not allowed to a thread while a capture in global mode is under way, unless the thread says that it
// knows what it is doing; neither touches the capturing stream.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

void CUDART_CB graph_block_released(void* b) { static_cast<GraphBlock*>(b)->released.store(true); }

void free_released_blocks() {
    for (auto it = graph_blocks.begin(); it != graph_blocks.end();) {
        if (!it->released.load()) { ++it; continue; }
        RelaxedCapture relaxed;
        cudaFree(it->p);
        it = graph_blocks.erase(it);
    }
}

bool graph_block(unsigned long long capture, cudaGraph_t graph, size_t bytes, Block* out) {
    GraphBlock* b = nullptr;
    for (GraphBlock& o : graph_blocks) if (!o.released.load() && o.capture == capture && o.bytes >= bytes) b = &o;
    if (!b) {
        for (GraphBlock& o : graph_blocks) if (o.released.load() && o.bytes >= bytes && (!b || o.bytes < b->bytes)) b = &o;
        if (!b) {
            void* p = nullptr;
            {
                RelaxedCapture relaxed;
                if (scratch_malloc(&p, COUNTER_BYTES + bytes) != cudaSuccess) return false;
            }
            graph_blocks.emplace_back();
            b = &graph_blocks.back();
            b->p = static_cast<uint8_t*>(p); b->bytes = bytes;
        }
        b->capture = capture;
        b->released.store(false);
        cudaUserObject_t owner;
        if (cudaUserObjectCreate(&owner, b, graph_block_released, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
            cudaGetLastError(); b->released.store(true); return false;
        }
        if (cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove) != cudaSuccess) {
            cudaGetLastError(); cudaUserObjectRelease(owner, 1); return false;          // (the release marks the block)
        }
        if (cudaMemsetAsync(b->p, 0, COUNTER_BYTES, g.stream) != cudaSuccess) { cudaGetLastError(); return false; }
    }
    out->p = b->p + COUNTER_BYTES; out->bytes = b->bytes; out->counters = reinterpret_cast<uint32_t*>(b->p);
    return true;
}

}  // namespace

bool launch_block(DevBuf& buf, size_t bytes, Block* out) {
    *out = Block{};
    out->counters = g.counters;
    if (bytes == 0) return true;
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long capture = 0;
    cudaGraph_t graph = nullptr;
    if (cudaStreamGetCaptureInfo(g.stream, &status, &capture, &graph) != cudaSuccess) cudaGetLastError();
    if (status == cudaStreamCaptureStatusActive) return graph_block(capture, graph, bytes, out);
    if (!graph_blocks.empty()) free_released_blocks();
    if (!buf.ensure(bytes)) return false;
    out->p = buf.p; out->bytes = buf.cap;
    return true;
}

// Scratch for a projection; where the memory is not to be had, by the rules that need the least.
bool workspace_for(qg::GemmArgs& a, qg::Workspace& ws) {
    Block b;
    if (!launch_block(g.ws_partial, qg::workspace_floats(a) * sizeof(float), &b)) {
        a.lean = 1;
        if (!launch_block(g.ws_partial, qg::workspace_floats(a) * sizeof(float), &b)) return false;
    }
    ws.partial = (float*)b.p; ws.partial_floats = b.bytes / sizeof(float);
    ws.counters = b.counters; ws.err = g.err_word;
    return true;
}

int validate_gemm(const void* X, size_t Xb, const void* W, size_t Wb, const void* Y, size_t Yb, int format, bool extended,
                  uint32_t M, uint32_t K, uint32_t N) {
    if (!g.initialized) return -1;
    if (!X || !W || !Y) return -2;
    if (((uintptr_t)X % 2 != 0) || ((uintptr_t)Y % 2 != 0)) return -2;
    const bool base_fmt = format >= 0 && format < 6;
    const bool ext_fmt = extended && (format == QUANT_PRISM_Q2_0 || format == QUANT_MLX_4BIT_G64 || format == QUANT_TERNARY_ROW ||
                                     format == QUANT_MLX_4BIT_PLANAR);
    if (!base_fmt && !ext_fmt) return -3;
    if (M == 0 || K == 0 || N == 0) return -4;
    if ((K % 32) != 0) return -4;
    if ((format == 2 || format == 4 || format == 5) && (K % 256) != 0) return -4;
    if (format == QUANT_PRISM_Q2_0 && (K % 128) != 0) return -4;
    if (format == QUANT_MLX_4BIT_G64 && (K % 64) != 0) return -4;
    const size_t min_x = (size_t)M * K * 2, min_y = (size_t)M * N * 2;
    const size_t min_w = compute_quant_matrix_bytes((QuantFormat)format, K, N);
    if (Xb < min_x || Yb < min_y || Wb < min_w) return -2;
    return 0;
}

int run_gemm(void* X, size_t Xb, void* W0, void* W1, size_t Wb, void* Y, size_t Yb, int format, uint32_t M, uint32_t K,
             uint32_t N, int layout, uint32_t H, uint32_t D, void* residual) {
    int rc = 0;
    const size_t x_bytes = (size_t)M * K * 2, y_bytes = (size_t)M * N * 2;
    const size_t w_bytes = compute_quant_matrix_bytes((QuantFormat)format, K, N);
    qg::GemmArgs a;
    memset(&a, 0, sizeof(a));
    a.format = format;
    // Host buffers go through one of two staging sets, uploads on the copy-in stream, the download on the
    // copy-out stream; consecutive calls alternate sets, so call i+1 uploads while call i computes and downloads.
    // The slot's buffers are reused two calls later: its uploads wait for the kernel that last read them, its
    // kernel waits for the download that last read its output buffer.
    StageSlot& sl = g.slots[g.slot_seq & 1u];
    bool staged_in = false;
    a.X = stage_in(X, x_bytes, sl, sl.x, false, &staged_in, &rc);
    if (rc) return rc;
    a.W0 = stage_in(W0, w_bytes, sl, sl.w0, true, &staged_in, &rc);
    if (rc) return rc;
    if (W1) { a.W1 = stage_in(W1, w_bytes, sl, sl.w1, true, &staged_in, &rc); if (rc) return rc; }
    if (residual) { a.residual = stage_in(residual, y_bytes, sl, sl.res, false, &staged_in, &rc); if (rc) return rc; }
    void* host_dst = nullptr;
    if (is_device_ptr(Y)) {
        a.Y = Y;
    } else {
        if (!sl.y.ensure(y_bytes)) return -5;
        a.Y = sl.y.p;
        host_dst = Y;
    }
    a.M = M; a.N = N; a.K = K; a.layout = layout; a.H = H; a.D = D;
    a.force_generic = g.force_generic;
    (void)Xb; (void)Wb; (void)Yb;
    qg::Workspace ws;
    if (!workspace_for(a, ws)) return -5;
    if (staged_in) {
        cudaEventRecord(sl.ev_in, g.stream_in);
        cudaStreamWaitEvent(g.stream, sl.ev_in, 0);
    }
    if (host_dst && sl.out_pending) cudaStreamWaitEvent(g.stream, sl.ev_out, 0);
    cudaError_t e = qg::launch(a, ws, g.stream);
    if (e != cudaSuccess) { set_error(std::string("kernel launch failed: ") + cudaGetErrorString(e)); return -6; }
    g.launches += (uint64_t)qg::last_launch_count();
    if (staged_in || host_dst) {
        cudaEventRecord(sl.ev_kernel, g.stream);
        sl.used = true;
        g.slot_seq++;
    }
    if (host_dst) {
        g.copies = true; g.copy_seq++;
        cudaStreamWaitEvent(g.stream_out, sl.ev_kernel, 0);
        if (cudaMemcpyAsync(host_dst, a.Y, y_bytes, cudaMemcpyDeviceToHost, g.stream_out) != cudaSuccess) { cudaGetLastError(); return -5; }
        cudaEventRecord(sl.ev_out, g.stream_out);
        sl.out_pending = true; sl.out_ptr = static_cast<const char*>(host_dst); sl.out_bytes = y_bytes;
        sl.out_seq = ++g.dispatch_seq;
        g.d2h_bytes += y_bytes;
    }
    return 0;
}

// Everything the bridge has enqueued, on all three streams (caller holds no lock-protected references).
cudaError_t sync_all_streams(cudaStream_t main, cudaStream_t in, cudaStream_t out) {
    cudaError_t e = cudaStreamSynchronize(in);
    cudaError_t e2 = cudaStreamSynchronize(main);
    cudaError_t e3 = cudaStreamSynchronize(out);
    return e != cudaSuccess ? e : (e2 != cudaSuccess ? e2 : e3);
}

}  // namespace bridge

using namespace bridge;

extern "C" {

int b200_bridge_error_seen = 0;

bool m4_bridge_init(const char*) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (g.initialized) return true;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        set_error("no CUDA device: this library has no CPU path");
        return false;
    }
    cudaGetDevice(&g.device);
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, g.device);
    if (prop.major != 10) {
        set_error("kernels are built for sm_100a only; found sm_" + std::to_string(prop.major) + std::to_string(prop.minor));
        return false;
    }
    if (cudaStreamCreateWithFlags(&g.stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&g.stream_in, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&g.stream_out, cudaStreamNonBlocking) != cudaSuccess) { cudaGetLastError(); return false; }
    bool ev_ok = cudaEventCreateWithFlags(&g.ev_main_d2h, cudaEventDisableTiming) == cudaSuccess &&
                 cudaEventCreateWithFlags(&g.ev_caller, cudaEventDisableTiming) == cudaSuccess;
    g.copies = false;
    for (StageSlot& sl : g.slots) {
        ev_ok = ev_ok && cudaEventCreateWithFlags(&sl.ev_in, cudaEventDisableTiming) == cudaSuccess &&
                cudaEventCreateWithFlags(&sl.ev_kernel, cudaEventDisableTiming) == cudaSuccess &&
                cudaEventCreateWithFlags(&sl.ev_out, cudaEventDisableTiming) == cudaSuccess;
        sl.used = false; sl.out_pending = false; sl.out_ptr = nullptr; sl.out_bytes = 0;
    }
    if (!ev_ok) { cudaGetLastError(); return false; }
    g.slot_seq = 0; g.main_d2h_pending = false;
    if (cudaMalloc(&g.counters, 4096 * sizeof(uint32_t) + 64) != cudaSuccess) { cudaGetLastError(); return false; }
    cudaMemsetAsync(g.counters, 0, 4096 * sizeof(uint32_t) + 64, g.stream);
    // (the error word lies in host memory that the GPU sees: reading it costs no copy)
    void *err_host = nullptr, *err_dev = nullptr;
    if (cudaHostAlloc(&err_host, 64, cudaHostAllocMapped) != cudaSuccess || cudaHostGetDevicePointer(&err_dev, err_host, 0) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    g.err_host = static_cast<int*>(err_host);
    *g.err_host = 0;
    b200_bridge_error_seen = 0;
    g.err_word = static_cast<int*>(err_dev);
    cudaStreamSynchronize(g.stream);
    // everything that makes the driver load code or reserve memory happens here, not in a later dispatch: the kernels'
    // shared-memory attributes (which load the module image) and the static scratch array of the allocation-free entry point
    if (qg::prepare_device() != cudaSuccess) { cudaGetLastError(); set_error("setting kernel attributes failed"); return false; }
    static_scratch_prepare(g.device);
    g.launches = 0; g.h2d_bytes = 0; g.d2h_bytes = 0; g.dispatch_seq = 0;
    g.initialized = true;
    return true;
}

size_t m4_bridge_get_expected_weight_bytes(int format, uint32_t K, uint32_t N) {
    if (format < 0 || format >= 6) return 0;
    return compute_quant_matrix_bytes((QuantFormat)format, K, N);
}

size_t b200_bridge_weight_bytes(int format, uint32_t K, uint32_t N) {
    if (!((format >= 0 && format < 6) || format == QUANT_PRISM_Q2_0 || format == QUANT_MLX_4BIT_G64 || format == QUANT_TERNARY_ROW ||
          format == QUANT_MLX_4BIT_PLANAR))
        return 0;
    return compute_quant_matrix_bytes((QuantFormat)format, K, N);
}

int m4_bridge_dispatch_gemm(void* X, size_t Xb, void* W, size_t Wb, void* Y, size_t Yb, int format, uint32_t M, uint32_t K,
                            uint32_t N) {
    std::lock_guard<std::mutex> lock(g.mu);
    int rc = validate_gemm(X, Xb, W, Wb, Y, Yb, format, false, M, K, N);
    if (rc) return rc;
    return run_gemm(X, Xb, W, nullptr, Wb, Y, Yb, format, M, K, N, LAYOUT_STANDARD, 0, 0, nullptr);
}

int m4_bridge_dispatch_gemv(void* x, size_t xb, void* W, size_t Wb, void* y, size_t yb, int format, uint32_t K, uint32_t N) {
    return m4_bridge_dispatch_gemm(x, xb, W, Wb, y, yb, format, 1, K, N);
}

int b200_bridge_dispatch_gemm_ex(void* X, size_t Xb, void* W, size_t Wb, void* Y, size_t Yb, int format, uint32_t M, uint32_t K,
                                 uint32_t N, int layout, uint32_t H, uint32_t D, void* residual, size_t residual_bytes) {
    std::lock_guard<std::mutex> lock(g.mu);
    int rc = validate_gemm(X, Xb, W, Wb, Y, Yb, format, true, M, K, N);
    if (rc) return rc;
    if (layout != LAYOUT_STANDARD && layout != LAYOUT_DIRECT_HEAD) return -4;
    if (layout == LAYOUT_DIRECT_HEAD && (H == 0 || D == 0 || (uint64_t)H * D != N)) return -4;
    if (residual) {
        if (layout != LAYOUT_STANDARD) return -4;
        if (((uintptr_t)residual % 2) != 0 || residual_bytes < (size_t)M * N * 2) return -2;
    }
    return run_gemm(X, Xb, W, nullptr, Wb, Y, Yb, format, M, K, N, layout, H, D, residual);
}

int b200_bridge_dispatch_swiglu(void* X, size_t Xb, void* Wg, void* Wu, size_t Wb, void* Out, size_t Ob, int format, uint32_t M,
                                uint32_t K, uint32_t F) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (g.initialized && !Wu) return -2;
    int rc = validate_gemm(X, Xb, Wg, Wb, Out, Ob, format, true, M, K, F);
    if (rc) return rc;
    return run_gemm(X, Xb, Wg, Wu, Wb, Out, Ob, format, M, K, F, LAYOUT_STANDARD, 0, 0, nullptr);
}

int b200_bridge_dispatch_gemm_grouped(const void* X, const void* const* W, void* const* Y, const uint32_t* N, uint32_t count,
                                      int format, uint32_t M, uint32_t K, int layout, uint32_t D) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (!g.initialized) return -1;
    if (!X || !W || !Y || !N || count < 1 || count > 3) return -2;
    if (format < 0 || format >= 6) return -3;
    if (M == 0 || K == 0 || (K % 256) != 0) return -4;
    if (layout != LAYOUT_STANDARD && layout != LAYOUT_DIRECT_HEAD) return -4;
    for (uint32_t i = 0; i < count; i++) {
        if (!W[i] || !Y[i] || !is_device_ptr(W[i]) || !is_device_ptr(Y[i])) return -2;
        if (N[i] == 0 || (layout == LAYOUT_DIRECT_HEAD && (D == 0 || N[i] % D != 0))) return -4;
    }
    if (!is_device_ptr(X)) return -2;
    qg::GemmArgs a;
    memset(&a, 0, sizeof(a));
    a.format = format; a.X = X; a.W0 = W[0]; a.Y = Y[0]; a.M = M; a.N = N[0]; a.K = K; a.layout = layout; a.D = D;
    a.H = layout == LAYOUT_DIRECT_HEAD ? N[0] / D : 0;
    a.n_extra = count - 1;
    for (uint32_t i = 1; i < count; i++) { a.W_extra[i - 1] = W[i]; a.Y_extra[i - 1] = Y[i]; a.N_extra[i - 1] = N[i]; }
    a.force_generic = g.force_generic;
    qg::Workspace ws;
    if (!workspace_for(a, ws)) return -5;      // few-token grouped launches split K
    cudaError_t e = qg::launch(a, ws, g.stream);
    if (e == cudaErrorInvalidValue) { cudaGetLastError(); return -4; }
    if (e != cudaSuccess) { set_error(std::string("kernel launch failed: ") + cudaGetErrorString(e)); return -6; }
    g.launches += (uint64_t)qg::last_launch_count();
    return 0;
}

int b200_bridge_dispatch_qkv_fused(const void* X, const void* Wq, const void* Wk, const void* Wv, void* Q, void* Kc, void* Vc, int format,
                                   uint32_t M, uint32_t K, uint32_t Hq, uint32_t Hkv, uint32_t D, float rope_theta, uint32_t pos0,
                                   int kv_q8_0, uint32_t kv_tokens) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (!g.initialized) return -1;
    if (!X || !Wq || !Wk || !Wv || !Q || !Kc || !Vc) return -2;
    const void* ptrs[7] = {X, Wq, Wk, Wv, Q, Kc, Vc};
    for (const void* q : ptrs) if (!is_device_ptr(q)) return -2;
    if (format < 0 || format >= 6) return -3;
    if (M == 0 || K == 0 || Hq == 0 || Hkv == 0 || (D != 64 && D != 128) || K % 256 != 0 || Hq % Hkv != 0) return -4;
    if (kv_tokens == 0) kv_tokens = M;
    if (kv_q8_0 ? ((uint64_t)pos0 + M > kv_tokens) : (pos0 != 0 && kv_tokens != M)) return -4;
    if (!kv_q8_0 && kv_tokens != M) return -4;                 // fp16 K/V come out as [Hkv][M][D] of this call only
    qg::GemmArgs a;
    memset(&a, 0, sizeof(a));
    a.format = format; a.X = X; a.W0 = Wq; a.Y = Q; a.M = M; a.N = Hq * D; a.K = K; a.layout = LAYOUT_DIRECT_HEAD; a.H = Hq; a.D = D;
    a.n_extra = 2; a.W_extra[0] = Wk; a.W_extra[1] = Wv; a.Y_extra[0] = Kc; a.Y_extra[1] = Vc; a.N_extra[0] = a.N_extra[1] = Hkv * D;
    const uint32_t rope = rope_theta > 0.0f ? 1u : 0u, q8 = kv_q8_0 ? 2u : 0u;
    a.post[0] = rope; a.post[1] = rope | q8; a.post[2] = q8;
    a.kv_tokens = kv_tokens; a.kv_pos0 = kv_q8_0 ? pos0 : 0u;
    if (rope) {
        // (cos, sin) of positions pos0 .. pos0 + M - 1, rebuilt only when the request changes
        if (g.rope_M != M || g.rope_D != D || g.rope_theta != rope_theta || g.rope_pos0 != pos0 || !g.rope_table.p) {
            cudaStreamSynchronize(g.stream);                  // the table may still be in use by the previous launch
            if (!g.rope_table.ensure((size_t)M * (D / 2) * 8)) return -5;
            if (lops::build_rope_table(g.rope_table.p, M, D, rope_theta, pos0, g.stream) != cudaSuccess) { cudaGetLastError(); return -6; }
            g.rope_M = M; g.rope_D = D; g.rope_theta = rope_theta; g.rope_pos0 = pos0;
            g.launches++;
        }
        a.rope_table = g.rope_table.p;
    }
    if (!a.post[0] && !a.post[1] && !a.post[2]) {}            // nothing to fuse: a plain grouped launch
    qg::Workspace ws;
    if (!workspace_for(a, ws)) return -5;
    cudaError_t e = qg::launch(a, ws, g.stream);
    if (e == cudaErrorInvalidValue) { cudaGetLastError(); return -4; }
    if (e != cudaSuccess) { set_error(std::string("kernel launch failed: ") + cudaGetErrorString(e)); return -6; }
    g.launches += (uint64_t)qg::last_launch_count();
    return 0;
}

int b200_bridge_register_weights(const void* host_ptr, size_t bytes) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (!g.initialized) return -1;
    if (!host_ptr || bytes == 0) return -2;
    if (is_device_ptr(host_ptr)) return 0;     // already resident
    auto it = g.registered.find(host_ptr);
    if (it != g.registered.end()) { cudaFree(it->second.dev); g.registered.erase(it); }
    void* dev = nullptr;
    if (cudaMalloc(&dev, bytes) != cudaSuccess) { cudaGetLastError(); return -5; }
    if (cudaMemcpyAsync(dev, host_ptr, bytes, cudaMemcpyHostToDevice, g.stream) != cudaSuccess) { cudaGetLastError(); cudaFree(dev); return -5; }
    cudaStreamSynchronize(g.stream);
    g.registered[host_ptr] = Registered{dev, bytes};
    return 0;
}

int b200_bridge_unregister_weights(const void* host_ptr) {
    std::lock_guard<std::mutex> lock(g.mu);
    auto it = g.registered.find(host_ptr);
    if (it == g.registered.end()) return -2;
    sync_all_streams(g.stream, g.stream_in, g.stream_out);
    cudaFree(it->second.dev);
    g.registered.erase(it);
    return 0;
}

void m4_bridge_synchronize(void) {
    // The lock is not held while waiting (dispatches from other threads may go on), so the "copy pending" marks may
    // only be cleared for copies that were already enqueued when the wait began: their events are recorded under the
    // lock before the wait and queried afterwards.  A copy enqueued by another thread in between keeps its mark.
    cudaStream_t s, si, so;
    uint64_t seq_before, copy_seq_before;
    bool copies;
    {
        std::lock_guard<std::mutex> lock(g.mu);
        if (!g.initialized) return;
        s = g.stream; si = g.stream_in; so = g.stream_out;
        seq_before = g.dispatch_seq;
        copies = g.copies; copy_seq_before = g.copy_seq;
    }
    // (callers that hand in device pointers never use the copy streams: one wait instead of three)
    cudaError_t e = copies ? sync_all_streams(s, si, so) : cudaStreamSynchronize(s);
    {
        std::lock_guard<std::mutex> lock(g.mu);
        if (g.initialized) {
            if (copies && g.copy_seq == copy_seq_before) g.copies = false;
            b200_bridge_error_seen = *g.err_host;
            for (StageSlot& sl : g.slots)
                if (sl.out_pending && (sl.out_seq <= seq_before || cudaEventQuery(sl.ev_out) == cudaSuccess)) {
                    sl.out_pending = false; sl.out_ptr = nullptr; sl.out_bytes = 0;
                }
            if (g.main_d2h_pending && (g.main_d2h_seq <= seq_before || cudaEventQuery(g.ev_main_d2h) == cudaSuccess))
                g.main_d2h_pending = false;
            cudaGetLastError();     // cudaErrorNotReady from a query is not an error
        }
    }
    if (e != cudaSuccess) {
        std::lock_guard<std::mutex> lock(g.mu);
        set_error(std::string("stream error: ") + cudaGetErrorString(e));
        fprintf(stderr, "[b200_bridge] %s\n", g.last_error.c_str());
    }
}

double m4_bridge_get_uma_footprint_mb(void) {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) { cudaGetLastError(); return 0.0; }
    return (double)(total_b - free_b) / (1024.0 * 1024.0);
}

bool m4_bridge_is_initialized(void) {
    std::lock_guard<std::mutex> lock(g.mu);
    return g.initialized;
}

void m4_bridge_shutdown(void) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (!g.initialized) return;
    sync_all_streams(g.stream, g.stream_in, g.stream_out);
    for (StageSlot& sl : g.slots) {
        sl.x.release(); sl.w0.release(); sl.w1.release(); sl.res.release(); sl.y.release();
        cudaEventDestroy(sl.ev_in); cudaEventDestroy(sl.ev_kernel); cudaEventDestroy(sl.ev_out);
        sl.ev_in = sl.ev_kernel = sl.ev_out = nullptr; sl.used = false; sl.out_pending = false;
    }
    cudaEventDestroy(g.ev_main_d2h); g.ev_main_d2h = nullptr;
    cudaEventDestroy(g.ev_caller); g.ev_caller = nullptr;
    cudaStreamDestroy(g.stream_in); cudaStreamDestroy(g.stream_out); g.stream_in = g.stream_out = nullptr;
    g.stage_x.release(); g.stage_w0.release(); g.stage_w1.release(); g.stage_y.release(); g.stage_res.release();
    g.stage_aux0.release(); g.stage_aux1.release(); g.stage_aux2.release();
    g.ws_partial.release();
    g.rope_table.release(); g.rope_M = g.rope_D = 0;
    g.attn_scratch.release();
    free_released_blocks();              // (graphs that are still there keep theirs)
    for (auto& kv : g.registered) cudaFree(kv.second.dev);
    g.registered.clear();
    cudaFree(g.counters); g.counters = nullptr;
    cudaFreeHost(const_cast<int*>(g.err_host)); g.err_host = nullptr; g.err_word = nullptr;
    cudaStreamDestroy(g.stream); g.stream = nullptr;
    static_scratch_forget();
    g.initialized = false;
}

/* What the bridge enqueues from here on waits on the GPU for everything `stream` (a cudaStream_t; NULL: the default stream)
 * holds now.  -6 if that is not possible (`stream` or one of the bridge's own is being captured: an edge from work outside the
 * capture would end it): wait on the host instead. */
int b200_bridge_wait_stream(void* stream) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (!g.initialized) return -1;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing((cudaStream_t)stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) { cudaGetLastError(); return -6; }
    {
        RelaxedCapture relaxed;         // (a query would end a capture in global mode that is under way on any stream)
        if (cudaStreamQuery((cudaStream_t)stream) == cudaSuccess) return 0;     // nothing to wait for: one call instead of three
        cudaGetLastError();
    }
    if (capturing(g.stream) || capturing(g.stream_in)) return -6;
    if (cudaEventRecord(g.ev_caller, (cudaStream_t)stream) != cudaSuccess || cudaStreamWaitEvent(g.stream, g.ev_caller, 0) != cudaSuccess ||
        cudaStreamWaitEvent(g.stream_in, g.ev_caller, 0) != cudaSuccess) {
        cudaGetLastError();
        return -6;
    }
    return 0;
}

int b200_bridge_project(void* stream, void* X, size_t Xb, void* W, size_t Wb, void* Y, size_t Yb, int format, uint32_t M, uint32_t K,
                        uint32_t N) {
    if (b200_bridge_wait_stream(stream) == -6) return 1;
    const int rc = m4_bridge_dispatch_gemm(X, Xb, W, Wb, Y, Yb, format, M, K, N);
    if (rc == 0) m4_bridge_synchronize();
    return rc;
}

int b200_bridge_device_error(void) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (!g.initialized) return -1;
    cudaStreamSynchronize(g.stream);
    return b200_bridge_error_seen = *g.err_host;
}

int b200_bridge_clear_device_error(void) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (!g.initialized) return -1;
    sync_all_streams(g.stream, g.stream_in, g.stream_out);
    // A split-K launch that gave up on a bounded wait leaves its tile counters part-way: they are cleared with the error word,
    // so the next split-K launch starts from zero again.
    *g.err_host = b200_bridge_error_seen = 0;
    return cudaMemset(g.counters, 0, 4096 * sizeof(uint32_t) + 64) == cudaSuccess ? 0 : -6;
}

/* Testing hook: allocations of scratch beyond `bytes` fail as if the GPU were full (0: no limit). */
void b200_bridge_debug_limit_scratch(size_t bytes) {
    std::lock_guard<std::mutex> lock(g.mu);
    g.scratch_limit = bytes;
}

/* Testing hook: writes `value` into split-K tile counter `index` (what an aborted split-K launch leaves behind). */
int b200_bridge_debug_set_tile_counter(uint32_t index, uint32_t value) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (!g.initialized) return -1;
    if (index >= 4096) return -2;
    cudaStreamSynchronize(g.stream);
    return cudaMemcpy(g.counters + index, &value, sizeof(uint32_t), cudaMemcpyHostToDevice) == cudaSuccess ? 0 : -6;
}

/* Device memory that captured graphs hold as scratch (what graphs that are gone have left is given back first). */
size_t b200_bridge_graph_scratch_bytes(void) {
    std::lock_guard<std::mutex> lock(g.mu);
    free_released_blocks();
    size_t n = 0;
    for (const GraphBlock& b : graph_blocks) n += COUNTER_BYTES + b.bytes;
    return n;
}

const char* b200_bridge_last_error_string(void) { return g.last_error.c_str(); }
uint64_t b200_bridge_kernel_launches(void) { return g.launches; }
void* b200_bridge_stream(void) { return (void*)g.stream; }
void b200_bridge_force_generic(int on) { g.force_generic = on; }
void b200_bridge_enable_small_kernel(int on) { qg::set_small_kernel_enabled(on); }
void b200_bridge_enable_pair_kernel(int on) { qg::set_pair_kernel_enabled(on != 0); }
int b200_bridge_last_launch_pair(void) { return qg::last_launch_pairs(); }

}  // extern "C"
