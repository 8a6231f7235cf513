// Causal attention on tensor memory, head dim 64 and 128, any group size up to 128, the key range split where that fills
// the GPU.
//
//   Q [Hq][M][D] fp16, K and V [Hkv][Mkv][D] fp16 (a Q8_0 cache is expanded once per call by dequant_q8_0_kernel; value =
//   fp16(q * d), the rounding of the reference's dequantize_q8_0), O [M][Hq*D] or [Hq][M][D] fp16.  Query row i sits at
//   position pos0 + i and attends keys 0 .. pos0 + i (brick4_attn_kernels.metal:573-911, unified_8b_kernels.metal:857-998).
//
// One CTA = one kv head x two query tiles of 128 rows; a tile packs BP = 128 / G neighbouring positions of the G query
// heads that share the kv head (row r = head r / BP, position r % BP), so that one decode token still fills G rows and no
// K or V tile is fetched twice for the same positions.
//
//   warps 0-3, 4-7   softmax of tile 0 / tile 1: thread = query row = tensor-memory lane.  Scores come out of tensor
//                    memory, P = 2^(s - m) goes back as fp16 into columns of its own, from where
//                    tcgen05.mma takes it as its A operand: P never passes through shared memory, a row's maximum and sum
//                    need no shuffle, no exchange and no CTA barrier.
//   warp 8           S(it) = Q.K(it)^T of both tiles; for 64-wide heads also O += P(it).V(it)
//   warp 10          O += P(it).V(it) for 128-wide heads
//   warp 9           TMA: the Q tiles, then K(0), K(1), V(0), K(2), V(1), ... through one ring of slots.
//
//   tensor memory    S0, S1, then P0, P1, O0 and O1 in the last 2 D columns.  A softmax warp frees its scores as soon as they are in
//                    registers (s_free), and the next step's are computed while it is at the exponentials; P is written, and O
//                    rescaled, once the PV of the step before has completed (pv_done).  Both fit beside each other with steps of 64
//                    keys for 128-wide heads, of 128 for 64-wide.  (With P over the front half of its scores, S(it + 1) waits for
//                    PV(it): 32 heads of 64 over 2048 tokens 37.0 us instead of 32.1.)
//
// What bounds it: 64-wide heads the softmax, two warps a scheduler at 2850 cycles per step of 128 keys and two tiles, of which the
// exponential unit needs 1536; 128-wide heads the MMAs of 64 keys (1280 cycles: score MMAs of 64 columns read their Q operand from
// shared memory for 48 cycles each) and the hand-overs between them, 1500.
// Every mbarrier wait is bounded; on expiry the CTA records a code, its roles run out on whatever is there, the result is not stored, and it
// leaves once its copies have landed.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "attention_ws.cuh"
#include "bridge_state.cuh"
#include "exp2_poly.cuh"
#include "ptx.cuh"

namespace attn {
namespace ws {

constexpr int ROWS = 128;                                // query rows of a tile
constexpr int SOFTMAX_THREADS = 256;
constexpr int ATOM = 128 * 128;                          // bytes of [128 query rows][64 fp16] in the 128-byte-swizzled layout
constexpr int MAX_SPLITS = 32;

// keys of a step: as many as tensor memory has columns for beside the two accumulators
__host__ __device__ constexpr uint32_t step_keys(uint32_t d) { return d == 128u ? 64u : 128u; }
// Steps after which the reference maximum of a row may lag.  Distance from 64 bits for 32 / 8 heads over 2048 tokens; the same with queries of
// twice the size; 8 / 2 heads, 256 tokens behind 7936:
//   lag from the first step on    2.60e-4  2.70e-4  2.92e-4      35.0 us for the first
//   after three exact steps       2.56e-4  2.58e-4  2.89e-4
//   after four                    2.55e-4  2.54e-4  2.87e-4      36.8 us
//   never                         2.53e-4  2.31e-4  2.86e-4
// A lag with steps of 128 keys, which results may not be further than: 2.58e-4, 2.64e-4, 2.88e-4.
constexpr uint32_t EXACT_STEPS = 4;
template <int D> struct Cfg {
    static constexpr int BK = (int)step_keys(D);
    // Score and value MMAs from a thread each, so that neither's waits leave the tensor pipe idle (128-wide heads, 32 / 8 over 2048 tokens
    // behind 8192, 274 -> 265 us), or from one in an order that keeps the tiles half a step apart where the softmax takes longer than
    // the MMAs (64-wide, 32 heads, 2048 tokens 31.3 against 33.9).
    static constexpr bool TWO = D == 128;
    static constexpr int THREADS = SOFTMAX_THREADS + (TWO ? 96 : 64);
    // Batches of 16 accumulator columns that a rescaling has under way together.  128-wide heads that follow the maximum rescale in most
    // of their 64-key steps: 24 / 8 heads, 2048 tokens behind 8192, 267 us with one, 260 with two.  Four take 162 registers instead of
    // 130, and no block of the next kernel fits beside this one (32 / 8 heads, 33 tokens behind 500, 9.9 -> 10.7).  64-wide heads have
    // no registers for a second.
    static constexpr int RESCALE = D == 128 ? 2 : 1;
    static constexpr int ATOMS = D / 64;
    static constexpr int TILE = ATOMS * ATOM;            // a query tile
    static constexpr int KV_ATOM = BK * 128, KV_TILE = ATOMS * KV_ATOM;      // a K or V tile: [BK keys][64 fp16] twice or once
    static constexpr int SLOTS = D == 128 ? 9 : 6;       // K and V tiles in flight
    static constexpr size_t USED = 1024 + (size_t)2 * TILE + (size_t)SLOTS * KV_TILE + 512;
    // At least 160 KB: the CTA holds all 512 tensor-memory columns, so no CTA of a neighbouring kernel that also holds some
    // (the projection kernels, 80 KB and more) may share its SM.
    static constexpr size_t SMEM = USED < 160 * 1024 ? 160 * 1024 : USED;
    // tensor-memory columns: scores of both tiles, probabilities (fp16 pairs) of both, accumulators of both
    static constexpr uint32_t COL_S = 0, COL_P = 2 * BK, COL_O = 512 - 2 * D;
    static_assert(3 * BK <= 512 - 2 * D, "scores, probabilities and accumulators fit tensor memory");
};

struct Params {
    __half* O;
    float* part_o;               // [split][Hq * M][D], unnormalised (split launches)
    float2* part_ml;             // [split][Hq * M]: reference maximum (log2 domain), sum
    uint32_t Hq, M, Mkv, pos0, G, BP, tiles_per_split;
    float scale_log2e;
    int out_tokens_major, split;
    uint32_t tiles;              // query tiles of a CTA (1 or 2)
    int* err;
};

// key tiles that the rows at positions [p, p + BP) of this call attend
template <int D> __device__ __forceinline__ uint32_t key_tiles(uint32_t p, uint32_t BP, uint32_t M, uint32_t Mkv, uint32_t pos0) {
    if (p >= M) return 0u;
    return min(pos0 + min(p + BP, M) - 1u, Mkv - 1u) / step_keys(D) + 1u;
}

__device__ __forceinline__ float ex2(float x) {           // 2^x, one instruction on the special-function unit; ex2(-inf) = 0
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// two fp32 values per instruction
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// 2^x of two values without the special-function unit: x = n + f with n the nearest integer (in the low mantissa bits of
// x + 1.5 * 2^23) and |f| <= 1/2, 2^f as a polynomial (exp2_poly.cuh), n added to the exponent field.  Inputs below
// -120 (masked scores are -inf) give 2^-120.  A NaN (the maximum propagates it) gives the largest fp32 number: infinite as a
// probability, and a sum that no row reaches otherwise (SUM_OF_NAN), by which the row is told to be NaN.  (Multiplying by 2^n instead
// keeps the NaN and costs 3 % of the 8B prefill.)
__device__ __forceinline__ float max_nan(float a, float b) {
    float y;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
    return y;
}
// a row's sum is at most 2^8 (see the lag) times 2^31 keys
constexpr float SUM_OF_NAN = 1e12f;
template <int DEG> __device__ __forceinline__ void ex2_poly2(float x0, float x1, float& e0, float& e1) {
    const uint64_t x = pack2(max_nan(x0, -120.0f), max_nan(x1, -120.0f));
    const uint64_t r = add2(x, pack2(12582912.0f, 12582912.0f));
    const uint64_t n = add2(r, pack2(-12582912.0f, -12582912.0f));
    const uint64_t f = fma2(n, pack2(-1.0f, -1.0f), x);
    uint64_t p = pack2(exp2poly::coef<DEG>(DEG), exp2poly::coef<DEG>(DEG));
#pragma unroll
    for (int i = DEG - 1; i >= 0; i--) p = fma2(p, f, pack2(exp2poly::coef<DEG>(i), exp2poly::coef<DEG>(i)));
    float p0, p1, r0, r1;
    unpack2(p, p0, p1);
    unpack2(r, r0, r1);
    e0 = __int_as_float(__float_as_int(p0) + (__float_as_int(r0) << 23));
    e1 = __int_as_float(__float_as_int(p1) + (__float_as_int(r1) << 23));
}
// How many pairs of eight, by what bounds the step: two for 64-wide heads, whose softmax follows the maximum exactly (32 heads, 2048 tokens:
// none 32.7 us, two 31.3, three 33.4), three for 128-wide heads with the lag (32 / 8 heads: none 35.5, two 35.1, three 33.3), none
// without it (24 / 8 heads, 1024 tokens: none 22.0, one 22.5).
template <int D, bool LAG> __device__ constexpr bool poly_pair(int j) {
    return D == 64 ? (j & 3) == 1 : LAG && ((j & 7) == 1 || (j & 7) == 4 || (j & 7) == 6);
}

__device__ __forceinline__ void tmem_ld_x32(uint32_t taddr, float* r) {
    uint32_t v[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) r[i] = __uint_as_float(v[i]);
}
__device__ __forceinline__ void tmem_st_x32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
          "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
          "r"(r[30]), "r"(r[31])
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]: fp16 operands, fp32 accumulate, A rows = lanes, two consecutive k per column
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// LAG: the reference maximum lags (see below) and the polynomial share of the exponentials is the short one
template <int D, bool LAG>
__global__ void __launch_bounds__(Cfg<D>::THREADS, 1)
attn_ws_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
               const Params p) {
    using C = Cfg<D>;
    constexpr int BK = C::BK;
    extern __shared__ uint8_t smem_raw_[];
    uint8_t* sQ = smem_raw_ + ((1024u - (ptx::smem_u32(smem_raw_) & 1023u)) & 1023u);    // [2 tiles]
    uint8_t* sKV = sQ + 2 * C::TILE;                                                      // [SLOTS]
    uint64_t* q_full = reinterpret_cast<uint64_t*>(sKV + C::SLOTS * C::KV_TILE);          // [2] query tile landed
    uint64_t* s_full = q_full + 2;                        // [2] scores of the step complete
    uint64_t* s_free = s_full + 2;                        // [2] ... and in registers: one arrival per softmax warp
    uint64_t* p_full = s_free + 2;                        // [2] probabilities written, O rescaled: one arrival per softmax warp
    uint64_t* pv_done = p_full + 2;                       // [2] O holds the step, the probabilities have been read
    uint64_t* kv_full = pv_done + 2;                      // [SLOTS]
    uint64_t* kv_empty = kv_full + C::SLOTS;              // [SLOTS]
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(kv_empty + C::SLOTS);
    volatile uint32_t* abort_flag = tmem_holder + 1;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // kv heads along x, position blocks along y, latest (longest) block first; splits of the key range along z
    const uint32_t hk = blockIdx.x;
    const uint32_t p0 = (gridDim.y - 1u - blockIdx.y) * p.tiles * p.BP;
    const uint32_t t0 = blockIdx.z * p.tiles_per_split;
    // steps of tile g inside this split
    auto steps_of = [&](uint32_t g) {
        if (g >= p.tiles) return 0u;
        const uint32_t n = key_tiles<D>(p0 + g * p.BP, p.BP, p.M, p.Mkv, p.pos0);
        return n > t0 ? min(n - t0, p.tiles_per_split) : 0u;
    };
    const uint32_t cnt0 = steps_of(0u), cnt1 = steps_of(1u);
    const uint32_t n_steps = max(cnt0, cnt1);
    if (n_steps == 0u) return;                            // this split lies behind the block's last key tile

    if (tid == SOFTMAX_THREADS + 32) {
        for (int i = 0; i < 2; i++) { ptx::mbar_init(&q_full[i], 1); ptx::mbar_init(&s_full[i], 1); ptx::mbar_init(&s_free[i], 4); ptx::mbar_init(&p_full[i], 4); ptx::mbar_init(&pv_done[i], 1); }
        for (int i = 0; i < C::SLOTS; i++) { ptx::mbar_init(&kv_full[i], 1); ptx::mbar_init(&kv_empty[i], 1); }
        *abort_flag = 0u;
        ptx::fence_barrier_init();
        ptx::prefetch_tensormap(&tmQ); ptx::prefetch_tensormap(&tmK); ptx::prefetch_tensormap(&tmV);
    }
    __syncwarp();
    if (warp == 8) { ptx::tmem_alloc(tmem_holder, 512); ptx::tmem_relinquish(); }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem = *tmem_holder;
    // everything above touched only this CTA's shared and tensor memory; global memory is first touched below
    ptx::grid_dependency_wait();
    ptx::launch_dependents();

    if (warp == 9) {
        // ---------------- copies: Q0, K(0), Q1, K(1), V(0), K(2), V(1), ... ----------------
        const uint32_t q_bytes = p.BP * p.G * 128u * (uint32_t)C::ATOMS;     // rows BP * G .. 127 of a tile stay unwritten: no output reads them
        auto load_q = [&](uint32_t g) {
            if (lane != 0u || (g ? cnt1 : cnt0) == 0u) return;
            ptx::mbar_arrive_expect_tx(&q_full[g], q_bytes);
            for (int a = 0; a < C::ATOMS; a++)
                ptx::tma_load_3d(sQ + g * C::TILE + a * ATOM, &tmQ, &q_full[g], a * 64, (int)(p0 + g * p.BP), (int)(hk * p.G));
        };
        load_q(0u);
        uint32_t slot = 0, ph = 0;
        bool ok = true;
        for (uint32_t i = 0; ok && i < 2u * n_steps; i++) {
            ok = __all_sync(0xffffffffu, ptx::mbar_wait(&kv_empty[slot], ph ^ 1u, abort_flag, p.err, 220));
            if (!ok) break;
            // i = 0: K(0); odd: the next K, or the last V; even: the V two steps behind it
            const bool is_k = i == 0u || ((i & 1u) && i + 1u < 2u * n_steps);
            const uint32_t step = i == 0u ? 0u : is_k ? (i + 1u) >> 1 : (i - 1u) >> 1;
            if (lane == 0) {
                ptx::mbar_arrive_expect_tx(&kv_full[slot], C::KV_TILE);
                for (int a = 0; a < C::ATOMS; a++)
                    ptx::tma_load_3d(sKV + slot * C::KV_TILE + a * C::KV_ATOM, is_k ? &tmK : &tmV, &kv_full[slot], a * 64, (int)((t0 + step) * BK), (int)hk);
            }
            if (i == 0u) load_q(1u);
            __syncwarp();
            if (++slot == (uint32_t)C::SLOTS) { slot = 0; ph ^= 1u; }
        }
    } else if (C::TWO && warp == 8) {
        // ---------------- scores: one thread, chosen once ----------------
        // The scores of a step are computed while the softmax of the step before is under way (it has moved its scores to registers), so they
        // are there when it ends.
        if (ptx::elect_one()) {
            const uint32_t idesc = ptx::umma_idesc_f16(128, BK);
            const uint64_t desc_hi = ptx::umma_desc_k_sw128(0u);
            const uint32_t q_lo = (ptx::smem_u32(sQ) & 0x3FFFFu) >> 4, kv_lo = (ptx::smem_u32(sKV) & 0x3FFFFu) >> 4;
            uint32_t slot = 0, ph = 0;                        // K(0), K(1), K(2), ... are copies 0, 1, 3, 5, ...
            for (uint32_t it = 0; it < n_steps; it++) {
                // (after a wait that gave up the rest runs out quickly, and nothing is written)
                ptx::mbar_wait(&kv_full[slot], ph, abort_flag, p.err, 221);
#pragma unroll
                for (uint32_t g = 0; g < 2u; g++) {
                    if (it >= (g ? cnt1 : cnt0)) continue;
                    if (it == 0u) ptx::mbar_wait(&q_full[g], 0u, abort_flag, p.err, 222);
                    else ptx::mbar_wait(&s_free[g], (it - 1u) & 1u, abort_flag, p.err, 225);
                    ptx::tc_fence_after_sync();
                    const uint64_t qd = desc_hi | (uint64_t)(q_lo + g * (C::TILE >> 4)), kd = desc_hi | (uint64_t)(kv_lo + slot * (C::KV_TILE >> 4));
#pragma unroll
                    for (int a = 0; a < C::ATOMS; a++)
#pragma unroll
                        for (int kk = 0; kk < 4; kk++)
                            ptx::umma_f16_ss(tmem + C::COL_S + g * BK, qd + a * (ATOM >> 4) + 2 * kk, kd + a * (C::KV_ATOM >> 4) + 2 * kk, idesc, (uint32_t)(a | kk) != 0u);
                    ptx::umma_commit(&s_full[g]);
                }
                ptx::umma_commit(&kv_empty[slot]);
                slot += it == 0u ? 1u : 2u;
                if (slot >= (uint32_t)C::SLOTS) { slot -= C::SLOTS; ph ^= 1u; }
            }
        }
        __syncwarp();
    } else if (C::TWO && warp == 10) {
        // ---------------- values: another thread, so that neither's waits leave the tensor pipe idle ----------------
        if (ptx::elect_one()) {
            const uint32_t idesc = ptx::umma_idesc_f16(128, D) | (1u << 16);          // B (= V) MN-major
            // V [key][d]: the 64 d of an atom row are the contiguous run, the second atom lies KV_ATOM bytes further (leading byte
            // offset), groups of eight keys are 1024 bytes apart (stride byte offset); 16 keys further = 2048 bytes
            const uint64_t vdesc_hi = ((uint64_t)(C::KV_ATOM >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
            const uint32_t kv_lo = (ptx::smem_u32(sKV) & 0x3FFFFu) >> 4;
            uint32_t slot = n_steps > 1u ? 2u : 1u, ph = 0;   // V(0), V(1), ... are copies 2, 4, ..., and the last one the copy behind its predecessor
            for (uint32_t it = 0; it < n_steps; it++) {
                ptx::mbar_wait(&kv_full[slot], ph, abort_flag, p.err, 223);
                const uint64_t vd = vdesc_hi | (uint64_t)(kv_lo + slot * (C::KV_TILE >> 4));
#pragma unroll
                for (uint32_t g = 0; g < 2u; g++) {
                    if (it >= (g ? cnt1 : cnt0)) continue;
                    ptx::mbar_wait(&p_full[g], it & 1u, abort_flag, p.err, 224);
                    ptx::tc_fence_after_sync();
#pragma unroll
                    for (int s = 0; s < BK / 16; s++)
                        umma_f16_ts(tmem + C::COL_O + g * D, tmem + C::COL_P + g * (BK / 2) + s * 8, vd + s * (2048 >> 4), idesc, (it | (uint32_t)s) != 0u);
                    ptx::umma_commit(&pv_done[g]);
                }
                ptx::umma_commit(&kv_empty[slot]);
                slot += it + 2u < n_steps ? 2u : 1u;
                if (slot >= (uint32_t)C::SLOTS) { slot -= C::SLOTS; ph ^= 1u; }
            }
        }
        __syncwarp();
    } else if (!C::TWO && warp == 8) {
        // ---------------- MMAs: one thread, chosen once ----------------
        // Tile 0 is half a step ahead of tile 1: S0(it + 1), P1(it - 1).V, S1(it + 1), P0(it).V.  The scores of a step are computed while the softmax
        // of the step before is under way (it has moved its scores to registers), so they are there when it ends.
        if (ptx::elect_one()) {
            const uint32_t idesc_s = ptx::umma_idesc_f16(128, BK);
            const uint32_t idesc_pv = ptx::umma_idesc_f16(128, D) | (1u << 16);       // B (= V) MN-major
            const uint64_t desc_hi = ptx::umma_desc_k_sw128(0u);
            // V [key][d]: the 64 d of an atom row are the contiguous run, the second atom lies KV_ATOM bytes further (leading byte
            // offset), groups of eight keys are 1024 bytes apart (stride byte offset); 16 keys further = 2048 bytes
            const uint64_t vdesc_hi = ((uint64_t)(C::KV_ATOM >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
            const uint32_t q_lo = (ptx::smem_u32(sQ) & 0x3FFFFu) >> 4, kv_lo = (ptx::smem_u32(sKV) & 0x3FFFFu) >> 4;
            // (after a wait that gave up the rest runs out quickly, and nothing is written)
            auto scores = [&](uint32_t g, uint32_t slot) {
                const uint64_t qd = desc_hi | (uint64_t)(q_lo + g * (C::TILE >> 4)), kd = desc_hi | (uint64_t)(kv_lo + slot * (C::KV_TILE >> 4));
#pragma unroll
                for (int a = 0; a < C::ATOMS; a++)
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)
                        ptx::umma_f16_ss(tmem + C::COL_S + g * BK, qd + a * (ATOM >> 4) + 2 * kk, kd + a * (C::KV_ATOM >> 4) + 2 * kk, idesc_s, (uint32_t)(a | kk) != 0u);
                ptx::umma_commit(&s_full[g]);
            };
            auto values = [&](uint32_t g, uint32_t slot, uint32_t it) {
                ptx::mbar_wait(&p_full[g], it & 1u, abort_flag, p.err, 224);
                ptx::tc_fence_after_sync();
                const uint64_t vd = vdesc_hi | (uint64_t)(kv_lo + slot * (C::KV_TILE >> 4));
#pragma unroll
                for (int s = 0; s < BK / 16; s++)
                    umma_f16_ts(tmem + C::COL_O + g * D, tmem + C::COL_P + g * (BK / 2) + s * 8, vd + s * (2048 >> 4), idesc_pv, (it | (uint32_t)s) != 0u);
                ptx::umma_commit(&pv_done[g]);
            };
            uint32_t slot = 0, ph = 0;                        // next slot of the ring, and its parity
            auto take_slot = [&](int code) {
                ptx::mbar_wait(&kv_full[slot], ph, abort_flag, p.err, code);
                const uint32_t r = slot;
                if (++slot == (uint32_t)C::SLOTS) { slot = 0; ph ^= 1u; }
                return r;
            };
            uint32_t k_slot = take_slot(221), v_slot = 0u, v_before = 0u;
#pragma unroll
            for (uint32_t g = 0; g < 2u; g++) {
                if ((g ? cnt1 : cnt0) == 0u) continue;
                ptx::mbar_wait(&q_full[g], 0u, abort_flag, p.err, 222);
                scores(g, k_slot);
            }
            ptx::umma_commit(&kv_empty[k_slot]);
            for (uint32_t it = 0; it <= n_steps; it++) {
                const bool more = it + 1u < n_steps;
                if (more) k_slot = take_slot(225);
                if (it + 1u < cnt0) {
                    ptx::mbar_wait(&s_free[0], it & 1u, abort_flag, p.err, 228);
                    ptx::tc_fence_after_sync();
                    scores(0u, k_slot);
                }
                if (it > 0u) {
                    if (it - 1u < cnt1) values(1u, v_before, it - 1u);
                    ptx::umma_commit(&kv_empty[v_before]);
                }
                if (it + 1u < cnt1) {
                    ptx::mbar_wait(&s_free[1], it & 1u, abort_flag, p.err, 229);
                    ptx::tc_fence_after_sync();
                    scores(1u, k_slot);
                }
                if (more) ptx::umma_commit(&kv_empty[k_slot]);
                if (it < n_steps) v_slot = take_slot(223);
                if (it < cnt0) values(0u, v_slot, it);
                v_before = v_slot;
            }
        }
        __syncwarp();
    } else if (warp < 8) {
        // ---------------- softmax ----------------
        const uint32_t g = warp >> 2;
        const uint32_t cnt = g ? cnt1 : cnt0;
        const uint32_t row = tid & 127u, hl = row / p.BP, pl = row - hl * p.BP;
        const uint32_t pos_first = p0 + g * p.BP, pos = pos_first + pl;
        const uint32_t last_key = min(p.pos0 + pos, p.Mkv - 1u);
        const uint32_t lane_addr = ((warp & 3u) * 32u) << 16;
        const uint32_t tS = tmem + lane_addr + C::COL_S + g * BK, tP = tmem + lane_addr + C::COL_P + g * (BK / 2), tOg = tmem + lane_addr + C::COL_O + g * D;
        // tiles whose keys all lie at or below every row's position (and inside the cache) need no mask
        const uint32_t free_keys = min(p.pos0 + pos_first + 1u, p.Mkv);
        float m_run = -1e30f, l_run = 0.0f;
        bool s_ready = false;
        for (uint32_t it = 0; it < cnt; it++) {
            // (after a wait that gave up the rest runs out quickly, and nothing is written)
            if (!s_ready) ptx::mbar_wait(&s_full[g], it & 1u, abort_flag, p.err, 226);
            __syncwarp();
            ptx::tc_fence_after_sync();
            const uint32_t k0 = (t0 + it) * BK;
            float sc[BK];
#pragma unroll
            for (int c = 0; c < BK; c += 32) tmem_ld_x32(tS + c, sc + c);
            ptx::tmem_ld_wait();
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s_free[g]);
            if (k0 + BK > free_keys) {
#pragma unroll
                for (int j = 0; j < BK; j++) if (k0 + j > last_key) sc[j] = -INFINITY;
            }
            float mx = -INFINITY, mx1 = -INFINITY;
#pragma unroll
            for (int j = 0; j < BK; j += 4) {
                mx = fmaxf(fmaxf(mx, sc[j]), sc[j + 1]);
                mx1 = fmaxf(fmaxf(mx1, sc[j + 2]), sc[j + 3]);
            }
            mx = fmaxf(mx, mx1) * p.scale_log2e;          // the scale is positive: max and scaling commute
            // With a lag of 8 the reference maximum moves only for jumps above 2^8: probabilities are then at most 256 instead of 1,
            // the division by the row sum removes the common factor, and O is rescaled hardly ever.  The first steps follow the maximum
            // exactly: the key that sets it has a probability of exactly 1, every other one is rounded, and the largest weigh most.
            float corr = 1.0f;
            if (mx > m_run + (LAG && it >= EXACT_STEPS ? 8.0f : 0.0f)) { corr = ex2(m_run - mx); m_run = mx; }
            const uint64_t sc2 = pack2(p.scale_log2e, p.scale_log2e), nm2 = pack2(-m_run, -m_run);
            uint64_t rs0 = 0ull, rs1 = 0ull;              // two zeros each
            // 64 keys at a time: exponentials, sums, and P as fp16 pairs.  Before the first of them is stored the step before has to be in O
            // and its probabilities read.
#pragma unroll
            for (int h = 0; h < BK / 64; h++) {
                const bool pv_ready = h == 0 && it > 0u ? ptx::mbar_test_wait(&pv_done[g], (it - 1u) & 1u) : true;
                uint32_t pk[32];
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const int e = h * 64 + 2 * j;
                    float x0, x1, e0, e1;
                    unpack2(fma2(pack2(sc[e], sc[e + 1]), sc2, nm2), x0, x1);     // masked: -inf stays -inf, 2^-inf = 0
                    if (poly_pair<D, LAG>(j)) ex2_poly2<LAG ? 5 : 6>(x0, x1, e0, e1);
                    else { e0 = ex2(x0); e1 = ex2(x1); }
                    if (j & 1) rs1 = add2(rs1, pack2(e0, e1)); else rs0 = add2(rs0, pack2(e0, e1));
                    pk[j] = pack_h2(e0, e1);
                }
                if (h == 0 && it > 0u) {
                    if (!pv_ready) ptx::mbar_wait(&pv_done[g], (it - 1u) & 1u, abort_flag, p.err, 227);
                    __syncwarp();
                    ptx::tc_fence_after_sync();
                    if (__any_sync(0xffffffffu, corr != 1.0f)) {
#pragma unroll
                        for (int c = 0; c < D; c += 16 * C::RESCALE) {
                            uint32_t v[C::RESCALE][16];
#pragma unroll
                            for (int b = 0; b < C::RESCALE; b++) ptx::tmem_ld_x16(tOg + c + 16 * b, v[b]);
                            ptx::tmem_ld_wait();
#pragma unroll
                            for (int b = 0; b < C::RESCALE; b++) {
#pragma unroll
                                for (int j = 0; j < 16; j++) v[b][j] = __float_as_uint(__uint_as_float(v[b][j]) * corr);
                                ptx::tmem_st_x16(tOg + c + 16 * b, v[b]);
                            }
                        }
                    }
                }
                tmem_st_x32(tP + h * 32, pk);
            }
            // (This look may park: what the warp does next is wait for these scores anyway, and P is on its way to tensor memory meanwhile.  One
            // that does not park, or stands behind the arrival below: 0 to 1 % slower, 2048 tokens of either head size.)
            s_ready = it + 1u < cnt && ptx::mbar_try_wait(&s_full[g], (it + 1u) & 1u);
            ptx::tmem_st_wait();
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&p_full[g]);
            float a0, a1;
            unpack2(add2(rs0, rs1), a0, a1);
            l_run = (l_run > SUM_OF_NAN ? l_run : l_run * corr) + (a0 + a1);
        }
        // ---------------- result ----------------
        if (cnt > 0u && __all_sync(0xffffffffu, ptx::mbar_wait(&pv_done[g], (cnt - 1u) & 1u, abort_flag, p.err, 227) && *abort_flag == 0u)) {
            ptx::tc_fence_after_sync();
            // Rows leave through the tile's Q buffer, which nothing reads any more: a thread deposits the 16-byte chunks of its
            // row (chunk c of row r at c ^ (r & 7): no bank conflict either way), then the warp moves its own 32 rows with whole
            // rows per store.  (Stores straight from the accumulator touch 32 rows each: about 4 us per CTA for fp32 partials.)
            constexpr uint32_t CH = D / 8;                           // chunks of a row per pass: D fp16, or D / 2 fp32
            const uint32_t head = hk * p.G + hl;
            const bool row_ok = hl < p.G && pos < p.M;
            const size_t r = (size_t)head * p.M + pos;
            const size_t split_row = (size_t)blockIdx.z * p.Hq * p.M + r;
            uint8_t* dst = p.split ? reinterpret_cast<uint8_t*>(p.part_o + split_row * D)
                                   : reinterpret_cast<uint8_t*>(p.O + (p.out_tokens_major ? ((size_t)pos * p.Hq + head) * D : r * D));
            if (!row_ok) dst = nullptr;
            if (p.split && row_ok) p.part_ml[split_row] = make_float2(m_run, l_run);
            const float inv = p.split ? 1.0f : (l_run > 0.0f && l_run <= SUM_OF_NAN ? 1.0f / l_run : 0.0f);      // (0: infinite O becomes NaN)
            uint8_t* stage = sQ + g * C::TILE;
            const uint32_t row0 = (warp & 3u) * 32u;
            const uint32_t cols = p.split ? D / 2u : (uint32_t)D;    // accumulator columns per pass
            for (uint32_t c0 = 0; c0 < (uint32_t)D; c0 += cols) {
                for (uint32_t c = 0; c < cols; c += 32u) {
                    float v[32];
                    tmem_ld_x32(tOg + c0 + c, v);
                    ptx::tmem_ld_wait();
                    if (p.split) {
#pragma unroll
                        for (uint32_t j = 0; j < 8u; j++)
                            *reinterpret_cast<float4*>(stage + row * (CH * 16u) + (((c / 4u + j) ^ (row & 7u)) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    } else {
#pragma unroll
                        for (uint32_t j = 0; j < 4u; j++)
                            *reinterpret_cast<uint4*>(stage + row * (CH * 16u) + (((c / 8u + j) ^ (row & 7u)) << 4)) =
                                make_uint4(pack_h2(v[8 * j] * inv, v[8 * j + 1] * inv), pack_h2(v[8 * j + 2] * inv, v[8 * j + 3] * inv),
                                           pack_h2(v[8 * j + 4] * inv, v[8 * j + 5] * inv), pack_h2(v[8 * j + 6] * inv, v[8 * j + 7] * inv));
                    }
                }
                __syncwarp();
                const uint32_t ch = lane % CH;
#pragma unroll 4
                for (uint32_t j = lane / CH; j < 32u; j += 32u / CH) {
                    uint8_t* d = reinterpret_cast<uint8_t*>(__shfl_sync(0xffffffffu, (unsigned long long)dst, (int)j));
                    const uint32_t rr = row0 + j;
                    const uint4 w = *reinterpret_cast<const uint4*>(stage + rr * (CH * 16u) + ((ch ^ (rr & 7u)) << 4));
                    if (d) *reinterpret_cast<uint4*>(d + c0 * 4u + ch * 16u) = w;        // (c0 > 0 only for fp32 rows)
                }
                __syncwarp();
            }
        }
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {      // let loads that are still in flight land before the CTA gives its shared memory back
        const long long c0 = clock64();
        while (clock64() - c0 < 4000000LL) { }
        __syncthreads();
    }
    if (warp == 8) { ptx::tc_fence_after_sync(); ptx::tmem_dealloc(tmem, 512); }
}

// Partial results of the splits of one row -> O: one warp per row, D / 32 values per lane.  The row's own tile says how many
// splits it has.
template <int D>
__global__ void __launch_bounds__(256) combine_kernel(const Params p) {
    ptx::grid_dependency_wait();
    ptx::launch_dependents();
    const uint32_t rows = p.Hq * p.M;
    const uint32_t r = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (r >= rows) return;
    const uint32_t head = r / p.M, pos = r - head * p.M;
    const uint32_t n = (key_tiles<D>(pos / p.BP * p.BP, p.BP, p.M, p.Mkv, p.pos0) + p.tiles_per_split - 1u) / p.tiles_per_split;
    // lane s holds split s's factor (at most 32 splits)
    const float2 ml = lane < n ? p.part_ml[(size_t)lane * rows + r] : make_float2(-1e30f, 0.0f);
    float m = ml.x;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float w = lane < n ? ex2(ml.x - m) : 0.0f;
    float l = ml.y > SUM_OF_NAN ? INFINITY : w * ml.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    const float wn = l > 0.0f ? w / l : 0.0f;
    constexpr int E = D / 32;
    float acc[E];
#pragma unroll
    for (int e = 0; e < E; e++) acc[e] = 0.0f;
    // eight splits' values are under way together
    const float* src = p.part_o + (size_t)r * D + lane * E;
    for (uint32_t s0 = 0; s0 < n; s0 += 8u) {
        float v[8][E];
#pragma unroll
        for (uint32_t j = 0; j < 8u; j++) {
            const float* at = src + (size_t)(s0 + j) * rows * D;
            if (s0 + j >= n) { for (int e = 0; e < E; e++) v[j][e] = 0.0f; }
            else if (E == 4) { const float4 t = __ldcg(reinterpret_cast<const float4*>(at)); v[j][0] = t.x; v[j][1] = t.y; v[j][E - 2] = t.z; v[j][E - 1] = t.w; }
            else { const float2 t = __ldcg(reinterpret_cast<const float2*>(at)); v[j][0] = t.x; v[j][1] = t.y; }
        }
#pragma unroll
        for (uint32_t j = 0; j < 8u; j++) {
            const float ws = __shfl_sync(0xffffffffu, wn, (int)(s0 + j));      // (lanes from n on hold 0: n is at most 32)
#pragma unroll
            for (int e = 0; e < E; e++) if (s0 + j < n) acc[e] = fmaf(ws, v[j][e], acc[e]);
        }
    }
    __half* dst = (p.out_tokens_major ? p.O + ((size_t)pos * p.Hq + head) * D : p.O + (size_t)r * D) + lane * E;
    if (E == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(pack_h2(acc[0], acc[1]), pack_h2(acc[E - 2], acc[E - 1]));
    else *reinterpret_cast<uint32_t*>(dst) = pack_h2(acc[0], acc[1]);
}

// Q8_0 records (34 bytes: fp16 d, 32 codes; 2-byte aligned) of K and then V -> fp16, value = fp16(q * d), one rounding.  Of the
// `total` records that the cache holds per kv head only the first `used` are expanded: those of the keys that some row sees (one
// token at position 4096 of a cache laid out for 32768, 8 heads of 128: 18 us instead of 58).  blockIdx.y walks over the heads
// of K and then of V.  A thread takes half a record (16 codes, two 16-byte stores); the integer becomes fp16 through the
// mantissa: 0x6400 | (q + 128) is 1152 + q.
constexpr uint32_t DEQUANT_THREADS = 256;
__global__ void __launch_bounds__(DEQUANT_THREADS) dequant_q8_0_kernel(const uint8_t* K, const uint8_t* V, __half* __restrict__ out,
                                                                       uint32_t heads, size_t total, size_t used) {
    ptx::grid_dependency_wait();
    ptx::launch_dependents();
    const size_t i = (size_t)blockIdx.x * DEQUANT_THREADS + threadIdx.x;
    const size_t b = i >> 1;
    if (b >= used) return;
    const __half2 off = __half2half2(__ushort_as_half((unsigned short)0x6480));      // 1152
    for (uint32_t h = blockIdx.y; h < 2u * heads; h += gridDim.y) {
        const uint16_t* blk = reinterpret_cast<const uint16_t*>((h < heads ? K + h * total * 34 : V + (h - heads) * total * 34) + b * 34);
        const uint16_t* c = blk + 1 + ((uint32_t)i & 1u) * 8u;
        uint16_t q[8];
#pragma unroll
        for (int e = 0; e < 8; e++) q[e] = ptx::ld(c + e);
        const __half2 d2 = __half2half2(__ushort_as_half(ptx::ld(blk)));
        uint32_t o[8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const uint32_t x = (__byte_perm((uint32_t)q[e], 0u, 0x4140u) ^ 0x00800080u) | 0x64006400u;
            const __half2 v = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&x), off), d2);
            o[e] = *reinterpret_cast<const uint32_t*>(&v);
        }
        uint4* dst = reinterpret_cast<uint4*>(out + (h * used + b) * 32 + ((uint32_t)i & 1u) * 16u);
        dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
        dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return (EncodeTiledFn)f;
    }();
    return fn;
}
// fp16 [heads][rows][D] as a 3-D map, boxes of box_heads x box_rows x 64 d with the 128-byte swizzle; rows past the end read as zero
bool make_map(CUtensorMap* m, const void* ptr, uint32_t D, uint32_t heads, uint32_t rows, uint32_t box_rows, uint32_t box_heads) {
    cuuint64_t dims[3] = {D, rows, heads};
    cuuint64_t strides[2] = {(cuuint64_t)D * 2, (cuuint64_t)rows * D * 2};
    cuuint32_t box[3] = {64, box_rows, box_heads};
    cuuint32_t estr[3] = {1, 1, 1};
    return encode_fn()(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

uint32_t sm_count() {
    static int n = 0;
    if (!n) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev); if (n <= 0) n = 148; }
    return (uint32_t)n;
}

// Query tiles of a CTA and splits of the key range, by estimated time.  The unit is a step of a CTA with two tiles: 64 keys of 128-wide
// heads or 128 keys of 64-wide ones.  One tile is cheaper a step and a CTA (FIXED), so one is taken while that leaves no more CTAs waiting
// for an SM.  Partial results cost a launch (COMBINE) and their way through memory (PER_BYTE).  One CTA runs per SM, so items beyond a whole
// number of waves cost a wave where all items are equally long (a chunk behind a long cache); a causal triangle from position 0 packs
// better than that, its sum is what counts there.
// The constants: least regret over 1050 shapes (1 to 1500 tokens behind 0 to 8192, 1 to 32 kv heads), each timed with every choice, with a
// penalty on choices worse than those of earlier constants: 1.4 % on average for 64-wide heads, 1.3 for 128-wide ones (0.7 where they follow
// the maximum exactly).
}  // namespace

// A lagging reference saves the rescaling of O and puts the result further from 64-bit arithmetic
// (EXACT_STEPS).  Results may not get less exact, so only the shapes whose results always had it have it.
static bool lagging(const Args& a) {
    const uint32_t G = a.Hq / a.Hkv;
    return a.D == 128 && (G == 1u || G == 2u || G == 4u || G == 8u);
}

Plan make_plan(const Args& a, bool split) {
    struct Model { float step[2], fixed[2], combine, per_byte; };
    static constexpr Model WIDE = {{0.829f, 1.0f}, {5.62f, 6.66f}, 3.86f, 0.387e-6f}, NARROW = {{0.921f, 1.0f}, {1.35f, 3.21f}, 2.63f, 0.349e-6f};
    static constexpr Model WIDE_EXACT = {{0.686f, 1.0f}, {0.97f, 0.9f}, 2.7f, 0.214e-6f};         // (heads that follow the maximum exactly)
    const Model& m = a.D == 64 ? NARROW : lagging(a) ? WIDE : WIDE_EXACT;
    const float (&STEP)[2] = m.step, (&FIXED)[2] = m.fixed, COMBINE = m.combine, PER_BYTE = m.per_byte;
    const float sms = (float)sm_count();
    Plan pl;
    pl.BP = (uint32_t)ROWS / (a.Hq / a.Hkv);
    auto key_tiles_at = [&](uint64_t pos) {      // key tiles of a block whose last position is `pos`
        const uint64_t last = (uint64_t)a.pos0 + (pos < a.M ? pos : a.M - 1);
        return (uint32_t)((last < a.Mkv - 1 ? last : a.Mkv - 1) / step_keys(a.D) + 1);
    };
    pl.n_last = key_tiles_at(a.M - 1);
    float best = 0.0f;
    pl.tiles = 0;
    for (uint32_t t = 2; t >= 1; t--) {
        const uint32_t blocks = (a.M + t * pl.BP - 1) / (t * pl.BP);
        if (t == 1u && blocks > 65535u) continue;
        const uint32_t n_first = key_tiles_at((uint64_t)t * pl.BP - 1);
        const bool even_lengths = 2u * n_first >= pl.n_last;
        for (uint32_t s = 1; s <= (split ? (uint32_t)MAX_SPLITS : 1u) && s <= pl.n_last; s++) {
            if (s > 2u && (float)a.Hkv * blocks * (s - 1) >= 2.0f * sms) break;        // the SMs are full without any more of them
            const uint32_t len = (pl.n_last + s - 1) / s;
            if ((pl.n_last + len - 1) / len != s) continue;                // the last split would be empty
            const float one = (float)len * STEP[t - 1] + FIXED[t - 1];
            float cost;
            if (even_lengths) {
                cost = ceilf((float)a.Hkv * blocks * s / sms) * one;
            } else {
                const float steps = (float)a.Hkv * blocks * 0.5f * (float)(n_first + pl.n_last);
                const float items = (float)a.Hkv * blocks * 0.5f * (float)((n_first + len - 1) / len + s);
                const float even = (steps * STEP[t - 1] + items * FIXED[t - 1]) / sms + 0.5f * (float)len * STEP[t - 1];
                cost = even > one ? even : one;
            }
            if (s > 1) cost += COMBINE + PER_BYTE * ((float)s * a.Hq * a.M * a.D * sizeof(float));
            if (pl.tiles == 0 || cost < best) { best = cost; pl.tiles = t; pl.blocks = blocks; pl.splits = s; }
        }
    }
    pl.kv_rows = a.pos0 + a.M < a.Mkv ? a.pos0 + a.M : a.Mkv;
    pl.kv_bytes = a.kv_fp16 ? 0 : (2 * (size_t)a.Hkv * pl.kv_rows * a.D * sizeof(__half) + 255) & ~(size_t)255;
    const size_t rows = pl.splits > 1 ? pl.splits * (size_t)a.Hq * a.M : 0;
    pl.o_bytes = rows * a.D * sizeof(float); pl.ml_bytes = rows * sizeof(float2);
    return pl;
}

namespace {

template <int D, bool LAG> cudaError_t launch_d(const Args& a, const Plan& planned, const Scratch& sc, cudaStream_t stream, int* launches) {
    using C = Cfg<D>;
    static std::atomic<uint64_t> attr_done{0};               // bit d: set on device d
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (!(attr_done.load() & bit)) {
        cudaError_t e = cudaFuncSetAttribute(attn_ws_kernel<D, LAG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        if (e != cudaSuccess) return e;
        attr_done |= bit;
    }
    const Plan pl = planned.scratch_bytes() <= sc.bytes ? planned : make_plan(a, false);
    if (pl.kv_bytes > sc.bytes) return cudaErrorMemoryAllocation;
    const uint32_t splits = pl.splits, blocks = pl.blocks;
    const size_t kv_bytes = pl.kv_bytes, o_bytes = pl.o_bytes, rows = (size_t)a.Hq * a.M;
    Params p;
    p.G = a.Hq / a.Hkv; p.BP = pl.BP;
    p.Hq = a.Hq; p.M = a.M; p.Mkv = a.Mkv; p.pos0 = a.pos0; p.scale_log2e = a.scale_log2e;
    p.out_tokens_major = a.out_tokens_major; p.O = (__half*)a.O; p.err = bridge::g.err_word;
    p.tiles_per_split = (pl.n_last + splits - 1) / splits;
    uint8_t* scratch = static_cast<uint8_t*>(sc.p);
    p.split = splits > 1; p.tiles = pl.tiles;
    p.part_o = reinterpret_cast<float*>(scratch + kv_bytes);
    p.part_ml = reinterpret_cast<float2*>(scratch + kv_bytes + o_bytes);

    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // a kernel's set-up may overlap the previous one's tail
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1; cfg.stream = stream;
    *launches = 0;
    const void *Kf = a.K, *Vf = a.V;
    if (!a.kv_fp16) {
        const size_t total = (size_t)a.Mkv * (D / 32), used = (size_t)pl.kv_rows * (D / 32);
        cfg.gridDim = dim3((unsigned)((2 * used + DEQUANT_THREADS - 1) / DEQUANT_THREADS), 2 * a.Hkv < 65535u ? 2 * a.Hkv : 65535u);
        cfg.blockDim = dim3(DEQUANT_THREADS);
        cudaError_t e = cudaLaunchKernelEx(&cfg, dequant_q8_0_kernel, (const uint8_t*)a.K, (const uint8_t*)a.V, (__half*)scratch, a.Hkv, total, used);
        if (e != cudaSuccess) return e;
        Kf = scratch; Vf = scratch + (size_t)a.Hkv * pl.kv_rows * D * sizeof(__half);
        ++*launches;
    }
    CUtensorMap tmQ, tmK, tmV;
    const uint32_t map_rows = a.kv_fp16 ? a.Mkv : pl.kv_rows;
    if (!make_map(&tmK, Kf, D, a.Hkv, map_rows, C::BK, 1) || !make_map(&tmV, Vf, D, a.Hkv, map_rows, C::BK, 1) || !make_map(&tmQ, a.Q, D, a.Hq, a.M, p.BP, p.G))
        return cudaErrorInvalidValue;
    cfg.gridDim = dim3(a.Hkv, blocks, splits); cfg.blockDim = dim3(C::THREADS); cfg.dynamicSmemBytes = C::SMEM;
    cudaError_t e = cudaLaunchKernelEx(&cfg, attn_ws_kernel<D, LAG>, tmQ, tmK, tmV, p);
    if (e != cudaSuccess) return e;
    ++*launches;
    if (splits > 1) {
        cfg.gridDim = dim3((unsigned)((rows + 7) / 8)); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = 0;
        e = cudaLaunchKernelEx(&cfg, combine_kernel<D>, p);
        if (e != cudaSuccess) return e;
        ++*launches;
    }
    return cudaSuccess;
}

}  // namespace

bool usable(const Args& a) {
    const uint32_t G = a.Hq / a.Hkv;
    if ((a.D != 64 && a.D != 128) || G > (uint32_t)ROWS || !(a.scale_log2e > 0.0f) || (((uintptr_t)a.Q | (uintptr_t)a.O) & 15u)) return false;
    if (a.kv_fp16 && (((uintptr_t)a.K | (uintptr_t)a.V) & 15u)) return false;
    // grid dimensions, 32-bit row and position arithmetic
    const uint32_t BP = (uint32_t)ROWS / G;
    if ((a.M + 2 * BP - 1) / (2 * BP) > 65535u || (uint64_t)a.pos0 + a.M > 0x7fffffffu || (uint64_t)a.Hq * a.M > 0x7fffffffu || a.Mkv > 0x7fffff00u) return false;
    return encode_fn() != nullptr;
}

cudaError_t launch(const Args& a, const Plan& plan, const Scratch& sc, cudaStream_t stream, int* launches) {
    if (a.D == 128) return lagging(a) ? launch_d<128, true>(a, plan, sc, stream, launches) : launch_d<128, false>(a, plan, sc, stream, launches);
    return launch_d<64, false>(a, plan, sc, stream, launches);
}

}  // namespace ws
}  // namespace attn
