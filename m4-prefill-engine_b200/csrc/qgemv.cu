// Single-token projection: the decode-like end of the path (m4_bridge_dispatch_gemv, and m4_bridge_dispatch_gemm with M = 1;
// reference: gemv_q4_0 and friends, quant_router_kernels.metal:930-1144).
//
// With one token the projection is a stream over the packed weights (9.4 MB at K = N = 4096) and what costs is instructions:
// unpacking a weight takes about two, and converting it to fp32, reading its activation and multiplying took three more.  Here
// the unpacked fp16 pairs go straight into warp-level MMAs (m16n8k16, fp32 accumulators): a warp works on 16 rows, lane 4 g + t
// on rows g and g + 8 with every fourth chunk of 256 elements.  The sum over K does not care about the order of K, so a lane's
// own pairs are the A fragment as they come out of the codec, and the B fragment is the activation pairs of the same elements
// (all eight columns alike); the MMA adds up the four lanes of a row.  The eight fragments' worth of K that one row's four lanes
// do not cover are other warps' chunks; they meet in shared memory.  (128-row tiles of tcgen05 would spend their time on
// latency here.  Q4_0 K = N = 4096, launches back to back: 8.1 us.  It was 6.1 while the weights were read in front of the wait for the launch before,
// which only callers that know who writes them may allow: early.)
// What bounds it: one dependent chain per warp (packed bytes, 2 x 4 x 130 instructions of unpacking at half rate, 64 MMAs) where the GPU
// has few warps, the unpack arithmetic where it has many (4096 -> 14336 13.8 us, 33 MB).
// Weights are those of the tensor-core kernels bit for bit (the same register-level codecs).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstring>

#include "codecs.cuh"
#include "ptx.cuh"
#include "qgemm.cuh"

namespace qg {

namespace {

constexpr int GV_MAX_WARPS = 8;
constexpr uint32_t X_CHUNK = 512 + 16;       // bytes of one activation chunk in shared memory: the four lanes of a row read
                                             // four neighbouring chunks at once, on different banks

struct GvParams {
    const __half* X; const uint8_t* W; __half* Y;
    uint32_t N, K, x_cols, x_wrap, chunks;       // chunks = K / 256; X has x_cols columns and starts over every x_wrap of K
    const uint8_t* meta;                     // planar layouts: scale / bias planes behind the packed plane
    const __half* row_scale;                 // per-row scale (integer-valued codecs)
    uint32_t early;                          // packed weights may be fetched before the preceding kernel has finished
};

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// bytes from one chunk to the next in a warp's buffer: an odd number of 16-byte pieces
__host__ __device__ constexpr uint32_t gv_stride(uint32_t rb) { return rb / 16u % 2u ? rb : rb + 16u; }

// R: rows per lane, 8 R rows per warp and CTA (R == 1 leaves the fragment's rows 8 .. 15 zero).
// STAGED: a warp's packed bytes pass through shared memory in the order in which they lie.  For chunks of 128 bytes: read by a lane each
// they lie at the same offset of 32 cache lines, on the same banks (group-64 layout, K = N = 4096 10.4 -> 8.2 us).  Elsewhere it
// costs what the copy takes (Q4_0 6.1 -> 7.1).
template <int FMT, int R, bool STAGED>
__global__ void __launch_bounds__(GV_MAX_WARPS * 32) qgemv_kernel(const GvParams p) {
    using Cd = cdc::Codec<FMT>;
    constexpr uint32_t ROWS = 8u * R;
    constexpr int RB = Cd::ROW_BYTES, MW = Cd::META_WORDS > 0 ? Cd::META_WORDS : 4;
    extern __shared__ __align__(16) uint8_t sx[];            // [chunks][X_CHUNK]
    __shared__ float part[GV_MAX_WARPS][ROWS];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, warps = blockDim.x >> 5;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const size_t row_bytes = (size_t)p.chunks * RB;
    const uint32_t n0 = blockIdx.x * ROWS;
    ptx::launch_dependents();
    if (!p.early) ptx::grid_dependency_wait();

    // (Ordinary loads, no __ldg: the launch in front may be writing what they read, a padded copy, and __ldg may be moved in front of the wait.)
    // packed bytes (and planar scales) of rows g, g + 8 and chunk c; rows past N repeat the last one, chunks past the end are zero
    uint32_t r[R][RB / 4], meta[R][MW];
    auto load = [&](uint32_t c, uint32_t (&r)[R][RB / 4], uint32_t (&meta)[R][MW]) {
#pragma unroll
        for (int h = 0; h < R; h++) {
            const uint32_t n = min(n0 + g + 8u * h, p.N - 1u);
            if (c < p.chunks) {
                if constexpr (!STAGED) {
                    const uint4* src = reinterpret_cast<const uint4*>(p.W + (size_t)n * row_bytes + (size_t)c * RB);
#pragma unroll
                    for (int i = 0; i < RB / 16; i++) {
                        const uint4 v = *(src + i);
                        r[h][4 * i] = v.x; r[h][4 * i + 1] = v.y; r[h][4 * i + 2] = v.z; r[h][4 * i + 3] = v.w;
                    }
                }
                if (Cd::META_WORDS != 0) {       // one scale and one bias per 64 (4 words) or 32 (8 words) elements, two planes
                    const uint32_t groups = (p.K / 256) * MW;
                    const uint8_t* mp = p.meta + ((size_t)n * groups + (size_t)c * MW) * 2;
                    const uint8_t* bp = mp + (size_t)p.N * groups * 2;
                    if (MW == 4) {
                        const uint2 sc = *reinterpret_cast<const uint2*>(mp), bi = *reinterpret_cast<const uint2*>(bp);
                        meta[h][0] = sc.x; meta[h][1] = sc.y; meta[h][2] = bi.x; meta[h][3] = bi.y;
                    } else {
                        const uint4 sc = *reinterpret_cast<const uint4*>(mp), bi = *reinterpret_cast<const uint4*>(bp);
                        meta[h][0] = sc.x; meta[h][1] = sc.y; meta[h][2] = sc.z; meta[h][3] = sc.w;
                        meta[h][MW - 4] = bi.x; meta[h][MW - 3] = bi.y; meta[h][MW - 2] = bi.z; meta[h][MW - 1] = bi.w;
                    }
                }
            } else {
                if constexpr (!STAGED) {
#pragma unroll
                    for (int i = 0; i < RB / 4; i++) r[h][i] = 0u;
                }
#pragma unroll
                for (int i = 0; i < MW; i++) meta[h][i] = 0u;
            }
        }
    };
    // STAGED: four chunks of the warp's rows, rows past N and chunks past the end as above, in its buffer
    constexpr uint32_t PIECES = RB / 16, STRIDE = gv_stride(RB);
    uint8_t* buf = sx + (size_t)p.chunks * X_CHUNK + (size_t)warp * (ROWS * 4u * STRIDE);
    auto fetch = [&](uint32_t c0) {
        const uint32_t dst = ptx::smem_u32(buf);
        static_assert(!STAGED || ROWS * 4u * PIECES % 32u == 0u, "whole turns of the warp");
#pragma unroll 3                                       // (all at once: 156 registers for 114, K = 14336 18.9 us for 16.9)
        for (uint32_t i = 0; i < ROWS * 4u * PIECES / 32u; i++) {
            const uint32_t j = i * 32u + lane, row = j / (4u * PIECES), k = j % (4u * PIECES), c = k / PIECES;
            const bool in = c0 + c < p.chunks;
            const uint8_t* src = in ? p.W + (size_t)min(n0 + row, p.N - 1u) * row_bytes + (size_t)c0 * RB + k * 16u : p.W;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (row * 4u + c) * STRIDE + (k - c * PIECES) * 16u), "l"(src), "r"(in ? 16 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if constexpr (STAGED) fetch(warp * 4u);
    load(warp * 4u + t, r, meta);                     // under way while the activations are staged
    if (p.early) ptx::grid_dependency_wait();

    // activations: fp16, columns past x_cols (of every period of x_wrap) are zero
    if ((reinterpret_cast<uintptr_t>(p.X) & 15u) == 0 && p.x_cols % 8u == 0u) {
        for (uint32_t i = tid; i < p.K / 8u; i += blockDim.x) {
            const uint32_t k = i * 8u, col = p.x_wrap == p.K ? k : k % p.x_wrap;
            const uint4 v = col < p.x_cols ? *reinterpret_cast<const uint4*>(p.X + col) : make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4*>(sx + (k >> 8) * X_CHUNK + (k & 255u) * 2u) = v;
        }
    } else {
        for (uint32_t k = tid; k < p.K; k += blockDim.x) {
            const uint32_t col = k % p.x_wrap;
            *reinterpret_cast<__half*>(sx + (k >> 8) * X_CHUNK + (k & 255u) * 2u) = col < p.x_cols ? p.X[col] : __half(0.0f);
        }
    }
    __syncthreads();

    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (uint32_t c0 = warp * 4u; c0 < p.chunks; c0 += warps * 4u) {
        const uint32_t c = c0 + t;
        // (a lane without a chunk multiplies what its codec makes of zero bytes, a finite number, with zeros)
        const uint8_t* xc = sx + (c < p.chunks ? c : 0u) * X_CHUNK;
        const uint32_t keep = c < p.chunks ? 0xffffffffu : 0u;
        // short rows leave the registers to fetch the next chunk while this one is multiplied
        constexpr bool AHEAD = RB <= 96 && Cd::META_WORDS == 0;
        const bool more = c0 + warps * 4u < p.chunks;
        uint32_t rn[AHEAD ? R : 1][AHEAD ? RB / 4 : 1], mn[AHEAD ? R : 1][AHEAD ? MW : 1];
        if constexpr (AHEAD) { if (more) load(c + warps * 4u, rn, mn); }
        if constexpr (STAGED) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();                             // every lane's copies are there
#pragma unroll
            for (int h = 0; h < R; h++)
#pragma unroll
                for (int i = 0; i < RB / 16; i++) {
                    const uint4 v = *reinterpret_cast<const uint4*>(buf + ((g + 8u * h) * 4u + t) * STRIDE + i * 16);
                    r[h][4 * i] = v.x; r[h][4 * i + 1] = v.y; r[h][4 * i + 2] = v.z; r[h][4 * i + 3] = v.w;
                }
            __syncwarp();                             // every lane has read: the next round may come while this one is multiplied
            if (more) fetch(c0 + warps * 4u);
        }
#pragma unroll
        for (int s = 0; s < 4; s++) {
            uint32_t a[R][32];
#pragma unroll
            for (int h = 0; h < R; h++) Cd::dequant64(r[h], s, a[h], meta[h]);
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const uint4 x = *reinterpret_cast<const uint4*>(xc + s * 128 + q * 16);
                mma16816(acc, a[0][4 * q], R == 2 ? a[R - 1][4 * q] : 0u, a[0][4 * q + 1], R == 2 ? a[R - 1][4 * q + 1] : 0u, x.x & keep, x.y & keep);
                mma16816(acc, a[0][4 * q + 2], R == 2 ? a[R - 1][4 * q + 2] : 0u, a[0][4 * q + 3], R == 2 ? a[R - 1][4 * q + 3] : 0u, x.z & keep, x.w & keep);
            }
        }
        if constexpr (AHEAD) {
            if (more) {
#pragma unroll
                for (int h = 0; h < R; h++)
#pragma unroll
                    for (int i = 0; i < RB / 4; i++) r[h][i] = rn[h][i];
            }
        } else if (more) load(c + warps * 4u, r, meta);
    }
    // every column of the accumulator is the same: rows g (acc[0]) and g + 8 (acc[2])
    if (t == 0u) { part[warp][g] = acc[0]; if (R == 2) part[warp][ROWS - 8u + g] = acc[2]; }
    __syncthreads();
    if (tid < ROWS && n0 + tid < p.N) {
        float sum = 0.0f;
        for (uint32_t w = 0; w < warps; w++) sum += part[w][tid];
        p.Y[n0 + tid] = __float2half_rn(Cd::ROW_SCALE ? sum * __half2float(p.row_scale[n0 + tid]) : sum);
    }
}

template <int FMT, int R, bool STAGED = false>
cudaError_t launch_gemv_rows(const GemmArgs& a, cudaStream_t stream) {
    using Cd = cdc::Codec<FMT>;
    GvParams p;
    p.X = (const __half*)a.X; p.W = (const uint8_t*)a.W0; p.Y = (__half*)a.Y;
    p.N = a.N; p.K = a.K; p.chunks = a.K / 256; p.x_cols = a.x_cols ? a.x_cols : a.K; p.x_wrap = a.x_wrap ? a.x_wrap : a.K;
    p.meta = (const uint8_t*)a.W0 + (size_t)a.N * p.chunks * Cd::ROW_BYTES;
    p.row_scale = (const __half*)p.meta;
    p.early = a.early_weights ? 1u : 0u;
    static std::atomic<uint64_t> attr_done{0};               // bit d: set on device d
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (!(attr_done.load() & bit)) {
        cudaError_t e = cudaFuncSetAttribute(qgemv_kernel<FMT, R, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) return e;
        attr_done |= bit;
    }
    const uint32_t groups = (p.chunks + 3u) / 4u;            // a warp takes four chunks at a time
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((a.N + 8 * R - 1) / (8 * R));
    const uint32_t rounds = (groups + GV_MAX_WARPS - 1) / GV_MAX_WARPS;
    cfg.blockDim = dim3(32u * ((groups + rounds - 1) / rounds));      // every warp the same number of rounds, as far as that goes
    static_assert(!STAGED || 199u * X_CHUNK + GV_MAX_WARPS * 8u * R * 4u * gv_stride(Cd::ROW_BYTES) <= 200u * 1024u, "activations and buffers of the longest rows");
    cfg.dynamicSmemBytes = (size_t)p.chunks * X_CHUNK + (STAGED ? (cfg.blockDim.x / 32u) * (8u * R * 4u * gv_stride(Cd::ROW_BYTES)) : 0u);
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, qgemv_kernel<FMT, R, STAGED>, p);
}

// SMs of the current device, asked of the runtime once for each
int gv_sms() {
    static std::atomic<int> known[64];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    const bool keep = dev >= 0 && dev < 64;
    if (keep && (n = known[dev].load()) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    if (keep) known[dev] = n;
    return n;
}

template <int FMT>
cudaError_t launch_gemv_fmt(const GemmArgs& a, cudaStream_t stream) {
    // Two rows per lane fill the fragment.  The variable-rate codec's two rows take 179 registers, one row 124 (K = 4096, N = 14336:
    // 31.3 against 23.5 us), and the codebook's 177 cost more than they give (K = N = 5120 18.3 against 11.6).
    constexpr bool ONE = FMT == QUANT_VAR_RATE_AFFINE || FMT == QUANT_EXL3, PLANAR = cdc::Codec<FMT>::META_WORDS != 0;
    if constexpr (ONE) return launch_gemv_rows<FMT, 1>(a, stream);
    else {
        // Where one row per lane makes less than a warp for each scheduler, the chain of one warp is the time, and half as long (K = N = 512:
        // Q4_K 3.9 -> 3.2 us, group-64 4.1 -> 3.3).  With 3.5 of them on an SM the formats that unpack fast lose 3 to 10 % (Q4_0 K = 512,
        // N = 4096 3.4 -> 3.7), the planar ones still gain 2 to 5 %.
        const uint32_t warps = (a.N + 7u) / 8u * ((a.K / 256u + 3u) / 4u);
        if (a.K / 256u <= 4u * GV_MAX_WARPS && warps <= (PLANAR ? 4u : 3u) * (uint32_t)gv_sms()) return launch_gemv_rows<FMT, 1>(a, stream);
        // (N = 5120: K = 512 4.7 us, staged 5.1; K = 1024 5.6 and 5.3)
        if constexpr (PLANAR) { if (a.K >= 1024u) return launch_gemv_rows<FMT, 2, true>(a, stream); }
        return launch_gemv_rows<FMT, 2>(a, stream);
    }
}

}  // namespace

bool gemv_path_ok(const GemmArgs& a) {
    if (a.force_generic || a.M != 1 || a.W1 || a.residual || a.partial_out || a.layout != 0 || a.scatter.world || a.n_extra) return false;
    if (a.K == 0 || a.K % 256 != 0 || a.N == 0) return false;
    if (((uintptr_t)a.W0 & 15u) || ((uintptr_t)a.X & 1u)) return false;
    if (a.K > 199u * 256u) return false;      // longer rows stay on the few-token kernel, as they always have (shared memory would hold twice that)
    switch (a.format) {
        case QUANT_Q4_0: case QUANT_MLX_4BIT: case QUANT_Q4_K: case QUANT_TERNARY_1_58: case QUANT_VAR_RATE_AFFINE: case QUANT_EXL3:
        case QUANT_MLX_4BIT_G64: case QUANT_TERNARY_ROW: case QUANT_MLX_4BIT_PLANAR: return true;
        default: return false;
    }
}

cudaError_t launch_gemv(const GemmArgs& a, cudaStream_t s) {
    switch (a.format) {
        case QUANT_Q4_0: return launch_gemv_fmt<QUANT_Q4_0>(a, s);
        case QUANT_MLX_4BIT: return launch_gemv_fmt<QUANT_MLX_4BIT>(a, s);
        case QUANT_Q4_K: return launch_gemv_fmt<QUANT_Q4_K>(a, s);
        case QUANT_TERNARY_1_58: return launch_gemv_fmt<QUANT_TERNARY_1_58>(a, s);
        case QUANT_VAR_RATE_AFFINE: return launch_gemv_fmt<QUANT_VAR_RATE_AFFINE>(a, s);
        case QUANT_EXL3: return launch_gemv_fmt<QUANT_EXL3>(a, s);
        case QUANT_MLX_4BIT_G64: return launch_gemv_fmt<QUANT_MLX_4BIT_G64>(a, s);
        case QUANT_MLX_4BIT_PLANAR: return launch_gemv_fmt<QUANT_MLX_4BIT_PLANAR>(a, s);
        case QUANT_TERNARY_ROW: return launch_gemv_fmt<QUANT_TERNARY_ROW>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace qg
