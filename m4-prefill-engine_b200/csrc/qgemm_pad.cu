// Packed weights with rows padded to whole chunks, for K that is not a multiple of the codecs' chunk (256 elements; 1024 for
// the 34-byte Prism blocks).
//
// The tensor-core kernels address packed rows through TMA maps, whose row stride has to be a multiple of 16 bytes: 18-byte
// Q4_0 blocks give that every 256 elements only.  One pass copies the rows into scratch at a chunk-aligned stride; what lies
// behind a row's last block is zero bytes, and the activation columns they meet read as zero (the map of X ends at the real
// K).
//
// The kernel that such shapes ran on (one thread per output, fp32) multiplied with weights that were never rounded to fp16,
// so the copy must not round them either.  A weight q * s (+ b) with a 4-bit q becomes a sum of terms that fp16 holds
// exactly: s = sh + sl, sh its leading 7 significant bits, sl the remaining 4, so that q * sh, q * sl and b are exact; the
// row holds the codes once per term with that term's scale and bias, and the activation columns start over for each.  Q4_0
// takes two terms, the affine formats three; ternary weights are exact as they are.  (Exact as long as every product is finite:
// outputs that come out infinite or NaN are computed again from the weights as they are, repair_nonfinite_kernel in qgemm.cu.)
//
// One launch in front, the packed bytes once or a few times more, and the repair pass behind: K = 2112, N = 1100, 129 tokens took
// 1707 us on the CUDA cores and takes 18 us, one token 336 and 13.  The CUDA-core kernel remains for activations that are not
// 16-byte aligned, for launches whose scratch has no room for the copy, and where the copy would be most of the work (pad_path_ok).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "../../include/quant_router.h"
#include "ptx.cuh"
#include "qgemm.cuh"

namespace qg {
namespace {

// A packed matrix is one to three planes of rows.  A plane is a run of records per row, `rec` bytes each, of which the 16-bit
// field at `scale_at` is a scale and the one at `bias_at` a bias (-1: none); the rest are codes.
struct Plane { uint64_t src, dst; uint32_t rows, src_row, dst_term; int32_t rec, scale_at, bias_at; };     // dst_term: bytes of one term of a padded row
struct Planes { Plane p[3]; uint32_t n, terms; uint64_t bytes; };

uint32_t padded_k(const GemmArgs& a) { const uint32_t c = chunk_elems(a.format); return (a.K + c - 1) / c * c; }

bool planes_of(const GemmArgs& a, Planes& out) {
    const uint64_t N = a.N;
    const uint32_t K = a.K, Kp = padded_k(a);
    memset(&out, 0, sizeof(out));
    out.terms = 1;
    auto add = [&](uint64_t src, uint32_t per, uint32_t rec, int scale_at, int bias_at) {      // one record of rec bytes per `per` elements
        out.p[out.n++] = Plane{src, out.bytes, a.N, K / per * rec, Kp / per * rec, (int32_t)rec, scale_at, bias_at};
        out.bytes += N * out.terms * (Kp / per * rec);
        return K % per == 0;
    };
    bool ok = true;
    switch (a.format) {
        case QUANT_Q4_0: out.terms = 2; ok = add(0, 32, 18, 0, -1); break;
        case QUANT_MLX_4BIT: out.terms = 3; ok = add(0, 32, 20, 0, 2); break;
        case QUANT_TERNARY_1_58: ok = add(0, 32, 12, -1, -1); break;
        case QUANT_PRISM_Q2_0: ok = add(0, 128, 34, -1, -1); break;
        case QUANT_MLX_4BIT_G64: {
            const uint64_t codes = N * (K / 2), plane = N * (K / 64) * 2;
            out.terms = 3;
            ok = add(0, 64, 32, -1, -1) && add(codes, 64, 2, 0, -1) && add(codes + plane, 64, 2, -1, 0);
            break;
        }
        case QUANT_MLX_4BIT_PLANAR: {
            const uint64_t n = N * (K / 32), scales = (n * 16 + 15) & ~(uint64_t)15, biases = (scales + n * 2 + 15) & ~(uint64_t)15;
            out.terms = 3;
            ok = add(0, 32, 16, -1, -1) && add(scales, 32, 2, 0, -1) && add(biases, 32, 2, -1, 0);
            break;
        }
        case QUANT_TERNARY_ROW:
            ok = add(0, 32, 8, -1, -1);
            // one scale per row, behind the codes: a single row of N scales, copied as it is
            out.p[out.n++] = Plane{N * (K / 4), out.bytes, 1u, a.N * 2u, a.N * 2u, 2, -1, -1};
            out.bytes += N * 2;
            break;
        default: return false;
    }
    out.bytes = (out.bytes + 255) & ~(uint64_t)255;
    return ok;
}

// bytes a thread writes at a time: rows and terms start on such a boundary (whole blocks and codes: 16; planes of scales: 8; the
// single row of per-row scales, whose length is N: 2)
__host__ __device__ inline uint32_t unit_of(const Plane& p) {
    return p.dst_term % 16u == 0u && p.dst % 16u == 0u ? 16u : (p.dst_term % 8u == 0u && p.dst % 8u == 0u ? 8u : 2u);
}

// scale of term t: leading 7 significant bits, the rest, nothing
__device__ __forceinline__ uint16_t scale_term(uint16_t bits, uint32_t t) {
    const bool finite = (bits & 0x7C00u) != 0x7C00u;
    const uint16_t hi = finite ? (uint16_t)(bits & 0xFFF0u) : bits;
    if (t == 0u) return hi;
    if (t == 1u && finite) return __half_as_ushort(__hsub(__ushort_as_half(bits), __ushort_as_half(hi)));      // exact
    return 0u;
}

// A thread owns UNIT bytes at one place of a padded row (plane blockIdx.z % n of matrix blockIdx.z / n) and walks down the rows:
// where it stands in a term, in a record and in its source row is worked out once.  Source rows are only 2-byte aligned in
// general; whole units come in with 4-byte loads, shifted by a half word where the row asks for it.
template <int UNIT>
__device__ __forceinline__ void pad_plane(const Plane& p, const uint8_t* src, uint8_t* dst, uint32_t terms) {
    constexpr int H = UNIT / 2;                                  // 16-bit fields per unit
    const uint32_t dst_row = p.dst_term * terms;
    const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) * UNIT;
    if (b >= dst_row) return;
    const uint32_t t = b / p.dst_term, off = b - t * p.dst_term;
    const uint32_t field0 = off % (uint32_t)p.rec;
    const bool whole = UNIT >= 8 && off + UNIT <= p.src_row;
    for (uint32_t row = blockIdx.y; row < p.rows; row += gridDim.y) {
        const uint8_t* s = src + (uint64_t)row * p.src_row + off;
        uint32_t v[(H + 1) / 2];
        const bool odd = (reinterpret_cast<uintptr_t>(s) & 2u) != 0;
        if (whole && !odd) {
#pragma unroll
            for (int i = 0; i < H / 2; i++) v[i] = ptx::ld(reinterpret_cast<const uint32_t*>(s) + i);
        } else if (whole && odd && (row > 0u || off > 0u) && (row + 1u < p.rows || off + UNIT + 2u <= p.src_row)) {
            // the words around it also hold the field before and the field behind, both inside the matrix
            uint32_t w[H / 2 + 1];
#pragma unroll
            for (int i = 0; i <= H / 2; i++) w[i] = ptx::ld(reinterpret_cast<const uint32_t*>(s - 2) + i);
#pragma unroll
            for (int i = 0; i < H / 2; i++) v[i] = __funnelshift_r(w[i], w[i + 1], 16);
        } else {
#pragma unroll
            for (int i = 0; i < (H + 1) / 2; i++) {
                const uint32_t o = off + 4u * i;
                const uint32_t lo = o < p.src_row ? *reinterpret_cast<const uint16_t*>(s + 4 * i) : 0u;
                const uint32_t hi = H > 1 && o + 2u < p.src_row ? *reinterpret_cast<const uint16_t*>(s + 4 * i + 2) : 0u;
                v[i] = lo | (hi << 16);
            }
        }
        if (terms > 1u) {
            int32_t field = (int32_t)field0;
#pragma unroll
            for (int e = 0; e < H; e++) {
                const uint32_t x = (v[e >> 1] >> (16 * (e & 1))) & 0xFFFFu;
                uint32_t y = x;
                if (field == p.scale_at) y = scale_term((uint16_t)x, t);
                if (field == p.bias_at && t + 1u != terms) y = 0u;
                v[e >> 1] ^= (x ^ y) << (16 * (e & 1));
                field += 2;
                if (field == p.rec) field = 0;
            }
        }
        uint8_t* d = dst + (uint64_t)row * dst_row + b;
        if constexpr (UNIT == 16) *reinterpret_cast<uint4*>(d) = make_uint4(v[0], v[1], v[2], v[3]);
        else if constexpr (UNIT == 8) *reinterpret_cast<uint2*>(d) = make_uint2(v[0], v[1]);
        else *reinterpret_cast<uint16_t*>(d) = (uint16_t)v[0];
    }
}

__global__ void __launch_bounds__(128) pad_rows_kernel(const uint8_t* w0, const uint8_t* w1, uint8_t* dst, const Planes pl) {
    ptx::launch_dependents();              // (the projection touches nothing before its own wait)
    ptx::grid_dependency_wait();           // the scratch may still be read by the launch before
    const uint32_t which = blockIdx.z % pl.n, matrix = blockIdx.z / pl.n;
    const Plane p = pl.p[which];
    const uint8_t* src = (matrix ? w1 : w0) + p.src;
    uint8_t* out = dst + matrix * pl.bytes + p.dst;
    if (unit_of(p) == 16u) pad_plane<16>(p, src, out, pl.terms);
    else if (unit_of(p) == 8u) pad_plane<8>(p, src, out, pl.terms);
    else pad_plane<2>(p, src, out, pl.terms);
}

}  // namespace

bool pad_path_ok(const GemmArgs& a) {
    if (a.force_generic || a.lean || a.x_cols || a.scatter.world || a.n_extra || a.wait_rows.flags || a.post[0] || a.post[1] || a.post[2]) return false;
    if (a.M == 0 || a.N == 0 || a.K == 0 || a.K % 8 != 0 || a.K % chunk_elems(a.format) == 0 || a.K > (1u << 24)) return false;
    if (((uintptr_t)a.X & 15u) || ((uintptr_t)a.W0 & 1u) || ((uintptr_t)a.W1 & 1u)) return false;
    // A single group of 64 padded to 256 and up to three terms is mostly copying: with few tokens the CUDA cores are done earlier (planar
    // formats, K = 64, N = 4096: 4 tokens 10.4 us against 20.9, 33 tokens 20.7 against 22.2, 129 tokens 55 against 22).
    if (a.K <= 64u && a.M <= 64u && (a.format == QUANT_MLX_4BIT_G64 || a.format == QUANT_MLX_4BIT_PLANAR || a.format == QUANT_TERNARY_ROW)) return false;
    Planes pl;
    return planes_of(a, pl);
}

void padded_shape(const GemmArgs& a, GemmArgs& padded) {
    Planes pl;
    planes_of(a, pl);
    padded.x_cols = a.K; padded.x_wrap = padded_k(a); padded.K = pl.terms * padded.x_wrap;
}

size_t padded_bytes(const GemmArgs& a) {
    Planes pl;
    return planes_of(a, pl) ? (size_t)pl.bytes * (a.W1 ? 2 : 1) : 0;
}

cudaError_t launch_pad(const GemmArgs& a, void* dst, GemmArgs& padded, cudaStream_t stream) {
    Planes pl;
    if (!planes_of(a, pl)) return cudaErrorInvalidValue;
    uint32_t across = 0, rows = 0;
    for (uint32_t i = 0; i < pl.n; i++) {
        const uint32_t units = (pl.p[i].dst_term * pl.terms + unit_of(pl.p[i]) - 1u) / unit_of(pl.p[i]);
        if (units > across) across = units;
        if (pl.p[i].rows > rows) rows = pl.p[i].rows;
    }
    padded = a;
    padded.early_weights = 0;                    // this kernel writes them
    padded_shape(a, padded);
    padded.W0 = dst;
    if (a.W1) padded.W1 = static_cast<uint8_t*>(dst) + pl.bytes;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    // one row per thread while that does not fill the GPU (148 SMs of 2048 threads), then up to eight
    const uint64_t fills = (uint64_t)across * rows / (148u * 2048u);
    const uint32_t per = fills < 1u ? 1u : (fills > 8u ? 8u : (uint32_t)fills);
    const uint32_t down = (rows + per - 1u) / per;
    cfg.gridDim = dim3((across + 127u) / 128u, down < 65535u ? down : 65535u, pl.n * (a.W1 ? 2u : 1u));
    cfg.blockDim = dim3(128);
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, pad_rows_kernel, (const uint8_t*)a.W0, (const uint8_t*)a.W1, (uint8_t*)dst, pl);
}

}  // namespace qg
