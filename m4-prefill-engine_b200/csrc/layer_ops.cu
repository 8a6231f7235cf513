// RMSNorm, rotary embedding and the fp32 residual add used by the decoder layer.
//
// The reference has these only in its Python block (src/engine/model.py:39-45 RMSNorm in its own
// code; :112-116 rotary embedding through a third-party array library, non-interleaved form), so
// the CPU oracle for them is a restatement (oracle/oracle.cpp: orc_rmsnorm, orc_rope).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>

#include "../../include/b200_bridge.h"
#include "bridge_state.cuh"
#include "layer_ops.cuh"
#include "ptx.cuh"

namespace lops {

// Every kernel of this file that a layer runs is launched so that its CTAs may be placed while the kernel in front of it
// drains (programmatic stream serialization); it touches memory only behind grid_dependency_wait, and lets the next kernel do
// the same from its own start.  The plain normalisation, which opens a layer, lets its successors be placed only once its own
// wait is over: from there on no kernel of the layer writes packed weights, and the projections may fetch theirs early.
template <class... P, class... A>
static cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, unsigned threads, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// One CTA of 256 threads per row, 8-element vectors.  Rows of up to KEEP * 2048 elements stay in registers between the sum and the
// scaling, and their weights are on the way during the reduction; longer rows are read a second time.
constexpr int KEEP = 4;
__device__ __forceinline__ void add_squares(float& ss, const uint4& v) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
    for (int j = 0; j < 4; j++) { const float2 f = __half22float2(h[j]); ss += f.x * f.x + f.y * f.y; }
}
__device__ __forceinline__ uint4 scale_row(const uint4& v, const uint4& w, float r) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
    const __half2* wh = reinterpret_cast<const __half2*>(&w);
    uint4 o;
    __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 f = __half22float2(h[j]), g = __half22float2(wh[j]);
        const __half2 n = __floats2half2_rn(f.x * r, f.y * r);          // rounded to fp16 first, as the reference does
        const float2 nf = __half22float2(n);
        oh[j] = __floats2half2_rn(nf.x * g.x, nf.y * g.y);
    }
    return o;
}

__global__ void __launch_bounds__(256) rmsnorm_kernel(const __half* X, const __half* __restrict__ W,
                                                      __half* __restrict__ Y, uint32_t K, float eps) {
    ptx::grid_dependency_wait();
    ptx::launch_dependents();
    const __half* x = X + (size_t)blockIdx.x * K;
    __half* y = Y + (size_t)blockIdx.x * K;
    float ss = 0.0f;
    const bool vec = (K % 8 == 0) && ((((uintptr_t)x | (uintptr_t)y | (uintptr_t)W) & 15u) == 0);
    const uint32_t nv = K / 8u;
    const bool keep = vec && nv <= (uint32_t)KEEP * 256u;
    uint4 xv[KEEP], wv[KEEP];
    if (keep) {
#pragma unroll
        for (int u = 0; u < KEEP; u++) {
            const uint32_t i = threadIdx.x + 256u * u;
            if (i < nv) xv[u] = reinterpret_cast<const uint4*>(x)[i];
        }
#pragma unroll
        for (int u = 0; u < KEEP; u++) {
            const uint32_t i = threadIdx.x + 256u * u;
            if (i < nv) wv[u] = reinterpret_cast<const uint4*>(W)[i];
        }
#pragma unroll
        for (int u = 0; u < KEEP; u++) if (threadIdx.x + 256u * u < nv) add_squares(ss, xv[u]);
    } else if (vec) {
        for (uint32_t i = threadIdx.x; i < nv; i += 256u) add_squares(ss, reinterpret_cast<const uint4*>(x)[i]);
    } else {
        for (uint32_t i = threadIdx.x; i < K; i += 256u) { float f = __half2float(x[i]); ss += f * f; }
    }
    __shared__ float red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) tot += red[i];
    const float r = 1.0f / sqrtf(tot / (float)K + eps);
    if (keep) {
#pragma unroll
        for (int u = 0; u < KEEP; u++) {
            const uint32_t i = threadIdx.x + 256u * u;
            if (i < nv) reinterpret_cast<uint4*>(y)[i] = scale_row(xv[u], wv[u], r);
        }
    } else if (vec) {
        for (uint32_t i = threadIdx.x; i < nv; i += 256u)
            reinterpret_cast<uint4*>(y)[i] = scale_row(reinterpret_cast<const uint4*>(x)[i], reinterpret_cast<const uint4*>(W)[i], r);
    } else {
        for (uint32_t i = threadIdx.x; i < K; i += 256u) {
            __half n = __float2half_rn(__half2float(x[i]) * r);
            y[i] = __float2half_rn(__half2float(n) * __half2float(W[i]));
        }
    }
}

__global__ void rope_kernel(__half* __restrict__ X, uint32_t M, uint32_t D, float log2_theta, uint32_t pos0, size_t total_pairs) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total_pairs) return;
    const uint32_t half = D / 2;
    const uint32_t j = (uint32_t)(i % half);
    const size_t row = i / half;                 // h*M + m
    const uint32_t m = (uint32_t)(row % M);
    const float inv_freq = exp2f(-2.0f * (float)j / (float)D * log2_theta);
    const float ang = (float)(pos0 + m) * inv_freq;
    float s, c;
    sincosf(ang, &s, &c);
    __half* x = X + row * D;
    const float a = __half2float(x[j]), b = __half2float(x[j + half]);
    x[j] = __float2half_rn(__fmaf_rn(a, c, -__fmul_rn(b, s)));
    x[j + half] = __float2half_rn(__fmaf_rn(b, c, __fmul_rn(a, s)));
}

// (cos, sin) of every (position, frequency) of a launch, for the projection epilogue that applies the rotation itself:
// table[m][j] = sincos((pos0 + m) * theta^(-2j/D)), the very expression of the kernels above, so a fused rotation and a
// separate one agree bit for bit.
__global__ void rope_table_kernel(float2* __restrict__ table, uint32_t M, uint32_t D, float log2_theta, uint32_t pos0) {
    const uint32_t half = D / 2;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)M * half) return;
    const uint32_t m = (uint32_t)(i / half), j = (uint32_t)(i % half);
    float s, c;
    sincosf((float)(pos0 + m) * exp2f(-2.0f * (float)j / (float)D * log2_theta), &s, &c);
    table[i] = make_float2(c, s);
}

// Rotate-half RoPE for D % 4 == 0: one thread owns two adjacent frequencies of one token and walks all heads, so
// the sine and cosine (the expensive part) are computed once per token and frequency instead of once per head, and
// every access is a 4-byte pair.  Element arithmetic is that of rope_kernel.
__global__ void rope_heads_kernel(__half* __restrict__ X, uint32_t H, uint32_t M, uint32_t D, float log2_theta, uint32_t pos0) {
    const uint32_t half = D / 2, per_tok = half / 2;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)M * per_tok) return;
    const uint32_t m = (uint32_t)(i / per_tok), j = 2u * (uint32_t)(i % per_tok);
    float s0, c0, s1, c1;
    sincosf((float)(pos0 + m) * exp2f(-2.0f * (float)j / (float)D * log2_theta), &s0, &c0);
    sincosf((float)(pos0 + m) * exp2f(-2.0f * (float)(j + 1) / (float)D * log2_theta), &s1, &c1);
    __half* x = X + (size_t)m * D + j;
    const size_t head_stride = (size_t)M * D;
    // heads in batches of four: all loads of a batch are issued before its first store (the stores would
    // otherwise order every later load behind them, one memory round trip per head)
    for (uint32_t h0 = 0; h0 < H; h0 += 4, x += 4 * head_stride) {
        __half2 lo[4], hi[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (h0 + u < H) {
                lo[u] = *reinterpret_cast<const __half2*>(x + u * head_stride);
                hi[u] = *reinterpret_cast<const __half2*>(x + u * head_stride + half);
            }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (h0 + u < H) {
                const float a0 = __low2float(lo[u]), a1 = __high2float(lo[u]), b0 = __low2float(hi[u]), b1 = __high2float(hi[u]);
                // (multiply-adds spelled out so that every kernel that rotates rounds alike)
                *reinterpret_cast<__half2*>(x + u * head_stride) =
                    __halves2half2(__float2half_rn(__fmaf_rn(a0, c0, -__fmul_rn(b0, s0))), __float2half_rn(__fmaf_rn(a1, c1, -__fmul_rn(b1, s1))));
                *reinterpret_cast<__half2*>(x + u * head_stride + half) =
                    __halves2half2(__float2half_rn(__fmaf_rn(b0, c0, __fmul_rn(a0, s0))), __float2half_rn(__fmaf_rn(b1, c1, __fmul_rn(a1, s1))));
            }
    }
}

__global__ void add_residual_f32_kernel(const __half* __restrict__ A, const float* __restrict__ B, __half* __restrict__ Y, size_t n) {
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i + 3 < n) {
        const float4 b = *reinterpret_cast<const float4*>(B + i);
        const __half2 a0 = *reinterpret_cast<const __half2*>(A + i), a1 = *reinterpret_cast<const __half2*>(A + i + 2);
        *reinterpret_cast<__half2*>(Y + i) = __floats2half2_rn(__low2float(a0) + b.x, __high2float(a0) + b.y);
        *reinterpret_cast<__half2*>(Y + i + 2) = __floats2half2_rn(__low2float(a1) + b.z, __high2float(a1) + b.w);
    } else {
        for (size_t k = i; k < n; k++) Y[k] = __float2half_rn(__half2float(A[k]) + B[k]);
    }
}

// Y = fp16(A + B), eight elements per thread (16-byte accesses; the launcher checks alignment and n % 8)
__global__ void add_residual_f16_kernel(const __half* __restrict__ A, const __half* __restrict__ B, __half* __restrict__ Y, size_t n8) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n8) return;
    const uint4 a = reinterpret_cast<const uint4*>(A)[i], b = reinterpret_cast<const uint4*>(B)[i];
    uint4 o;
    const __half2* ah = reinterpret_cast<const __half2*>(&a);
    const __half2* bh = reinterpret_cast<const __half2*>(&b);
    __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 fa = __half22float2(ah[j]), fb = __half22float2(bh[j]);
        oh[j] = __floats2half2_rn(fa.x + fb.x, fa.y + fb.y);
    }
    reinterpret_cast<uint4*>(Y)[i] = o;
}

// Residual add fused into the normalisation that follows it: S = fp16(A + B) (the block's output, kept for the next
// residual), Y = rmsnorm(S) * W.  One CTA of 256 threads per row; a thread reads back only the vectors it wrote itself,
// and the barrier of the row reduction separates every read of A from the first write of Y, so Y may alias A.
// Rows must be 16-byte aligned with K a multiple of 8 (checked by the launcher).
__global__ void __launch_bounds__(256) rmsnorm_add_kernel(const __half* A, const __half* B,
                                                          const __half* __restrict__ W, __half* __restrict__ S, __half* Y,
                                                          uint32_t K, float eps) {
    ptx::launch_dependents();
    ptx::grid_dependency_wait();
    const size_t row = (size_t)blockIdx.x * K;
    const uint32_t nv = K / 8u;
    const bool keep = nv <= (uint32_t)KEEP * 256u;
    float ss = 0.0f;
    auto add = [](const uint4& a, const uint4& b) {
        const __half2* ah = reinterpret_cast<const __half2*>(&a);
        const __half2* bh = reinterpret_cast<const __half2*>(&b);
        uint4 o;
        __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 fa = __half22float2(ah[j]), fb = __half22float2(bh[j]);
            oh[j] = __floats2half2_rn(fa.x + fb.x, fa.y + fb.y);
        }
        return o;
    };
    uint4 sv[KEEP], bv[KEEP];
    if (keep) {
#pragma unroll
        for (int u = 0; u < KEEP; u++) {
            const uint32_t i = threadIdx.x + 256u * u;
            if (i < nv) { sv[u] = reinterpret_cast<const uint4*>(A + row)[i]; bv[u] = reinterpret_cast<const uint4*>(B + row)[i]; }
        }
#pragma unroll
        for (int u = 0; u < KEEP; u++) {
            const uint32_t i = threadIdx.x + 256u * u;
            if (i < nv) {
                sv[u] = add(sv[u], bv[u]);
                add_squares(ss, sv[u]);
                reinterpret_cast<uint4*>(S + row)[i] = sv[u];
                bv[u] = reinterpret_cast<const uint4*>(W)[i];           // the weights, during the reduction
            }
        }
    } else {
        for (uint32_t i = threadIdx.x; i < nv; i += 256u) {
            const uint4 o = add(reinterpret_cast<const uint4*>(A + row)[i], reinterpret_cast<const uint4*>(B + row)[i]);
            add_squares(ss, o);
            reinterpret_cast<uint4*>(S + row)[i] = o;
        }
    }
    __shared__ float red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) tot += red[i];
    const float r = 1.0f / sqrtf(tot / (float)K + eps);
    if (keep) {
#pragma unroll
        for (int u = 0; u < KEEP; u++) {
            const uint32_t i = threadIdx.x + 256u * u;
            if (i < nv) reinterpret_cast<uint4*>(Y + row)[i] = scale_row(sv[u], bv[u], r);
        }
    } else {
        for (uint32_t i = threadIdx.x; i < nv; i += 256u)
            reinterpret_cast<uint4*>(Y + row)[i] = scale_row(reinterpret_cast<const uint4*>(S + row)[i], reinterpret_cast<const uint4*>(W)[i], r);
    }
}

cudaError_t rmsnorm(const void* X, const void* weight, void* Y, uint32_t M, uint32_t K, float eps, cudaStream_t s) {
    return launch_pdl(rmsnorm_kernel, dim3(M), 256, s, (const __half*)X, (const __half*)weight, (__half*)Y, K, eps);
}
cudaError_t rmsnorm_add(const void* A, const void* B, const void* weight, void* S, void* Y, uint32_t M, uint32_t K, float eps,
                        cudaStream_t s) {
    if (K % 8 != 0 || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(weight) |
                        reinterpret_cast<uintptr_t>(S) | reinterpret_cast<uintptr_t>(Y)) & 15u))
        return cudaErrorInvalidValue;
    return launch_pdl(rmsnorm_add_kernel, dim3(M), 256, s, (const __half*)A, (const __half*)B, (const __half*)weight, (__half*)S, (__half*)Y, K, eps);
}
cudaError_t rope(void* X, uint32_t H, uint32_t M, uint32_t D, float theta, uint32_t pos0, cudaStream_t s) {
    if (D % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 3u) == 0) {
        const size_t threads = (size_t)M * (D / 4);
        rope_heads_kernel<<<(unsigned)((threads + 127) / 128), 128, 0, s>>>((__half*)X, H, M, D, log2f(theta), pos0);
        return cudaGetLastError();
    }
    const size_t pairs = (size_t)H * M * (D / 2);
    rope_kernel<<<(unsigned)((pairs + 255) / 256), 256, 0, s>>>((__half*)X, M, D, log2f(theta), pos0, pairs);
    return cudaGetLastError();
}
// Everything between the Q/K/V projections and attention in one pass: rotary embedding on Q and K (in place for Q),
// K and V compressed to Q8_0 records and overwritten by the values those give back.  A warp takes one token and one batch of
// four rows -- four Q heads, or K and V of two kv heads (blockIdx.y: first the batches of Q, then those of K and V) -- so
// that its four loads are in flight together and a 33-token launch still has a hundred CTAs.  (One warp per token walking all
// heads was a chain of memory latencies: 16.4 us between events for 33 tokens of the 8B shape, 7.2 now; 20.5 -> 16.4 for 2048.)  Lane l holds elements E l .. E l + E - 1 of a row, E = D / 32;
// the rotation partner (i +- D/2) sits 16 lanes away and the 32 values of a Q8_0 record are those of 32 / E neighbouring lanes.
// Arithmetic is that of rope_heads_kernel and of attn::quantize_q8_0_kernel, bit for bit.
template <int D>
__global__ void __launch_bounds__(128) kv_post_kernel(__half* Q, __half* K, __half* V, uint8_t* __restrict__ Kq, uint8_t* __restrict__ Vq,
                                                      const float2* __restrict__ table, uint32_t Hq, uint32_t Hkv, uint32_t M, int rope, int q8, int dq) {
    constexpr int E = D / 32, W = E / 2;          // elements and 32-bit words per lane
    ptx::launch_dependents();
    ptx::grid_dependency_wait();
    const uint32_t m = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (m >= M) return;
    const uint32_t q_batches = rope ? (Hq + 3u) / 4u : 0u;
    const bool is_q = blockIdx.y < q_batches;
    // row u of the batch: its head, and the matrix it belongs to
    uint32_t head[4];
    __half* base[4];
    bool on[4];
#pragma unroll
    for (uint32_t u = 0; u < 4u; u++) {
        head[u] = is_q ? blockIdx.y * 4u + u : (blockIdx.y - q_batches) * 2u + (u >> 1);
        base[u] = is_q ? Q : ((u & 1u) ? V : K);
        on[u] = head[u] < (is_q ? Hq : Hkv);
    }
    uint32_t w[4][W];
#pragma unroll
    for (int u = 0; u < 4; u++)
        if (on[u]) {
            const __half* src = base[u] + ((size_t)head[u] * M + m) * D + lane * E;
            if (W == 2) { const uint2 t = *reinterpret_cast<const uint2*>(src); w[u][0] = t.x; w[u][W - 1] = t.y; }
            else w[u][0] = *reinterpret_cast<const uint32_t*>(src);
        }
    const bool upper = lane >= 16u;
    float2 cs[E];
    if (rope) {
        const float4* t4 = reinterpret_cast<const float4*>(table + (size_t)m * (D / 2) + (lane & 15u) * E);
#pragma unroll
        for (int e = 0; e < W; e++) { const float4 t = __ldg(t4 + e); cs[2 * e] = make_float2(t.x, t.y); cs[2 * e + 1] = make_float2(t.z, t.w); }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (!on[u]) continue;                     // (the same for every lane of the warp)
        const bool is_v = !is_q && (u & 1);
        __half* dst = base[u] + ((size_t)head[u] * M + m) * D + lane * E;
        if (rope && !is_v) {
            uint32_t r[W];
#pragma unroll
            for (int i = 0; i < W; i++) {
                const uint32_t pw = __shfl_xor_sync(0xffffffffu, w[u][i], 16);
                const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&w[u][i])), y = __half22float2(*reinterpret_cast<const __half2*>(&pw));
                const float2 c0 = cs[2 * i], c1 = cs[2 * i + 1];
                // lower half: a*c - b*s with (a, b) = (x, y); upper half: b*c + a*s with (a, b) = (y, x)
                const float r0 = upper ? __fmaf_rn(x.x, c0.x, __fmul_rn(y.x, c0.y)) : __fmaf_rn(x.x, c0.x, -__fmul_rn(y.x, c0.y));
                const float r1 = upper ? __fmaf_rn(x.y, c1.x, __fmul_rn(y.y, c1.y)) : __fmaf_rn(x.y, c1.x, -__fmul_rn(y.y, c1.y));
                const __half2 h = __floats2half2_rn(r0, r1);
                r[i] = *reinterpret_cast<const uint32_t*>(&h);
            }
#pragma unroll
            for (int i = 0; i < W; i++) w[u][i] = r[i];
        }
        bool write = rope && !is_v;
        if (!is_q && q8) {
            float v[E], amax = 0.0f;
#pragma unroll
            for (int i = 0; i < W; i++) { const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[u][i])); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
#pragma unroll
            for (int e = 0; e < E; e++) amax = fmaxf(amax, fabsf(v[e]));
#pragma unroll
            for (int o = 1; o < 32 / E; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            const float d = __fdiv_rn(amax, 127.0f);
            const float id = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
            const uint32_t part = lane % (32u / E);          // this lane's place in its record
            uint16_t* o = reinterpret_cast<uint16_t*>((is_v ? Vq : Kq) + (((size_t)head[u] * M + m) * (D / 32) + lane / (32u / E)) * 34u);
            const __half dh = __float2half_rn(d);
            if (part == 0u) o[0] = __half_as_ushort(dh);
#pragma unroll
            for (int i = 0; i < W; i++) {
                int q0 = (int)roundf(__fmul_rn(v[2 * i], id)), q1 = (int)roundf(__fmul_rn(v[2 * i + 1], id));
                q0 = max(-128, min(127, q0)); q1 = max(-128, min(127, q1));
                o[1u + part * W + i] = (uint16_t)((uint32_t)(uint8_t)(int8_t)q0 | ((uint32_t)(uint8_t)(int8_t)q1 << 8));
                w[u][i] = (uint32_t)__half_as_ushort(__hmul(__int2half_rn(q0), dh)) | ((uint32_t)__half_as_ushort(__hmul(__int2half_rn(q1), dh)) << 16);
            }
            write = dq;
        }
        if (write) {
            if (W == 2) *reinterpret_cast<uint2*>(dst) = make_uint2(w[u][0], w[u][W - 1]);
            else *reinterpret_cast<uint32_t*>(dst) = w[u][0];
        }
    }
}

cudaError_t kv_post(void* Q, void* K, void* V, void* Kq, void* Vq, const void* rope_table, uint32_t Hq, uint32_t Hkv,
                    uint32_t M, uint32_t D, bool rope, bool q8, bool dequant_in_place, cudaStream_t s) {
    if ((D != 64 && D != 128) || (rope && !rope_table) || (q8 && (!Kq || !Vq))) return cudaErrorInvalidValue;
    if (((reinterpret_cast<uintptr_t>(Q) | reinterpret_cast<uintptr_t>(K) | reinterpret_cast<uintptr_t>(V)) & 7u) ||
        (reinterpret_cast<uintptr_t>(rope_table) & 15u))
        return cudaErrorInvalidValue;
    const uint32_t batches = (rope ? (Hq + 3) / 4 : 0) + (Hkv + 1) / 2;
    if (batches > 65535u) return cudaErrorInvalidValue;
    return launch_pdl(D == 128 ? kv_post_kernel<128> : kv_post_kernel<64>, dim3((M + 3) / 4, batches), 128, s, (__half*)Q, (__half*)K, (__half*)V,
                      (uint8_t*)Kq, (uint8_t*)Vq, (const float2*)rope_table, Hq, Hkv, M, rope ? 1 : 0, q8 ? 1 : 0, (q8 && dequant_in_place) ? 1 : 0);
}

cudaError_t build_rope_table(void* table, uint32_t M, uint32_t D, float theta, uint32_t pos0, cudaStream_t s) {
    const size_t n = (size_t)M * (D / 2);
    rope_table_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>((float2*)table, M, D, log2f(theta), pos0);
    return cudaGetLastError();
}
cudaError_t add_residual_f32(const void* A, const float* B, void* Y, size_t n, cudaStream_t s) {
    const size_t threads = (n + 3) / 4;
    add_residual_f32_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>((const __half*)A, B, (__half*)Y, n);
    return cudaGetLastError();
}

cudaError_t add_residual_f16(const void* A, const void* B, void* Y, size_t n, cudaStream_t s) {
    if (n % 8 != 0 || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(Y)) & 15u))
        return cudaErrorInvalidValue;
    const size_t n8 = n / 8;
    add_residual_f16_kernel<<<(unsigned)((n8 + 255) / 256), 256, 0, s>>>((const __half*)A, (const __half*)B, (__half*)Y, n8);
    return cudaGetLastError();
}

}  // namespace lops

using namespace bridge;

extern "C" {

int b200_bridge_rmsnorm(void* X, void* weight, void* Y, uint32_t M, uint32_t K, float eps) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (!g.initialized) return -1;
    if (!X || !weight || !Y) return -2;
    if (M == 0 || K == 0) return -4;
    int rc = 0;
    const size_t bytes = (size_t)M * K * 2;
    const void* x = resolve_in(X, bytes, g.stage_x, false, &rc);
    if (rc) return rc;
    const void* w = resolve_in(weight, (size_t)K * 2, g.stage_aux0, false, &rc);
    if (rc) return rc;
    void* host_dst = nullptr;
    void* y = resolve_out(Y, bytes, g.stage_y, &host_dst, &rc);
    if (rc) return rc;
    if (lops::rmsnorm(x, w, y, M, K, eps, g.stream) != cudaSuccess) return -6;
    g.launches++;
    if (host_dst && copy_back(host_dst, y, bytes) != 0) return -5;
    return 0;
}

/* In-place rotary embedding on X [H][M][D] (device or host pointer). */
int b200_bridge_rope(void* X, uint32_t H, uint32_t M, uint32_t D, float theta, uint32_t pos0) {
    std::lock_guard<std::mutex> lock(g.mu);
    if (!g.initialized) return -1;
    if (!X) return -2;
    if (H == 0 || M == 0 || D == 0 || (D % 2) != 0 || theta <= 0.0f) return -4;
    const size_t bytes = (size_t)H * M * D * 2;
    if (is_device_ptr(X)) {
        if (lops::rope(X, H, M, D, theta, pos0, g.stream) != cudaSuccess) return -6;
        g.launches++;
        return 0;
    }
    int rc = 0;
    void* x = const_cast<void*>(resolve_in(X, bytes, g.stage_x, false, &rc));
    if (rc) return rc;
    if (lops::rope(x, H, M, D, theta, pos0, g.stream) != cudaSuccess) return -6;
    g.launches++;
    return copy_back(X, x, bytes);
}

}  // extern "C"
