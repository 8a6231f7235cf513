// Few-token projection: Y[m][n] = sum_k X[m][k] * dequant(W)[n][k] for up to 128 tokens (the decode-like shapes M = 33 /
// 127 / 128 of the router sweep, bench_universal_router.mm:764-773, and every projection of a short prefill: up to three
// matrices in one launch, and the dual gate / up projection with SwiGLU), and for more where a long K has few tiles (small_path_ok).  HBM-bound: the packed weights are
// read once, so what matters is how fast an SM turns packed bytes into MMA operands.
//
// Differences from the persistent kernel in qgemm.cu, all aimed at that:
//   * the unpacked weights never touch shared memory: a thread owns one weight row = one tensor-memory lane, unpacks 64
//     elements to 32 registers of fp16 pairs and writes them with one tcgen05.st into a ring of A-operand stages in
//     tensor memory; the MMA takes A from tensor memory (tcgen05.mma [d], [a], b-desc) and only the activations from
//     shared memory.  That removes the 16 KB store + 16 KB operand read per 64-element step that bound the other kernel;
//   * small CTAs (4 unpack warps = the 4 lane quadrants, two copy warps, an MMA warp; <= 112 KB of shared memory, 256
//     tensor-memory columns) so that two CTAs share an SM and one's copies and unpacking overlap the other's;
//   * weights and activations of a step share a ring stage with one full and one empty barrier (128 elements of K; 64 for Prism): a wait costs
//     the issuing thread more than the four MMAs of 48 tokens behind it (100 cycles);
//   * one work item per CTA: K is split up to eight ways and the splits of a tile form a thread-block cluster.  Every CTA
//     writes its partial tile to a scratch buffer (which stays in L2), one cluster barrier later each CTA of the cluster
//     sums one slice of the token columns in split order -- deterministic -- and writes fp16 Y: no counters, no CTA that
//     has to add everything alone.  (Passing the partial tiles through distributed shared memory instead measured
//     slower: remote shared-memory stores ran at about 10 bytes per clock per SM.)
//
// Every mbarrier wait is bounded (ptx::mbar_wait).  The cluster barrier is a hardware barrier: every thread of every
// CTA reaches it on every path, including after a wait has given up.
//
// What bounds it: the unpack arithmetic.  Half-precision and logic instructions issue every other cycle, Q4_0 takes 64 and 48 of them
// for 64 weights and a warp 255 cycles; a 128 x 64 step takes an SM 281 cycles (two CTAs), where HBM would need 196.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>
#include <utility>

#include "codecs.cuh"
#include "ptx.cuh"
#include "qgemm.cuh"

namespace qg {
namespace small {

constexpr int W_TILE = 128;          // weight rows per tile = UMMA M = tensor-memory lanes
constexpr int KSTEP = 64;            // K elements per sub-tile (4 MMAs of K = 16)
constexpr int SUB_COLS = KSTEP / 2;  // fp16 pairs: 32 tensor-memory columns per sub-tile
// Sub-tiles per operand stage: one hand-over for two of them (33 tokens, K = 14336, N = 4096 17.3 -> 15.9 us), except where two stages
// of twice the activations do not fit beside two packed stages (the 272-byte rows)
template <int FMT> struct Ring {
    static constexpr int SPS = cdc::Codec<FMT>::CHUNK == 256 ? 2 : 1, A_COLS = SPS * SUB_COLS;
};
constexpr int TMEM_COLS = 256;       // accumulator (T columns), then the A ring
constexpr int MAX_RAW_STAGES = 6, MAX_STAGES = 7;     // ring depths are chosen per launch (stages_for)
constexpr int UNPACK_WARPS = 4;      // one per lane quadrant (one warp of each of the two CTAs keeps a scheduler's pipes 90 % busy: a second
                                     // group, 33 tokens, K = 14336 16.2 -> 16.6 us)
constexpr int THREADS = (UNPACK_WARPS + 3) * 32;    // warps 0-3 unpack + epilogue, then packed-weight copies, activation copies, MMAs
constexpr int RAW_WARP = UNPACK_WARPS, ACT_WARP = UNPACK_WARPS + 1, MMA_WARP = UNPACK_WARPS + 2;
constexpr int MAX_T = 128;
constexpr int GATE_ROWS = W_TILE / 2;    // SwiGLU tile: 64 gate rows and the same 64 up rows
constexpr size_t SMEM_LIMIT = 112 * 1024; // two CTAs per SM

// Development aid: with -DQS_TRACE the first CTA records clock64() stamps at its synchronisation points into a device
// array that b200_debug_small_trace copies out.  Compiled out otherwise.
#ifdef QS_TRACE
__device__ unsigned long long g_qs_trace[8][64];
#define QST(role, slot) do { if (blockIdx.x == QS_TRACE && (slot) < 64) g_qs_trace[role][slot] = clock64(); } while (0)
#else
#define QST(role, slot) do { } while (0)
#endif

// (in the order in which a launch needs them, 64 bytes to a line of the constant cache, which is cold when a CTA starts)
struct Params {
    uint32_t n_w_tiles, k_splits, split_shift, chunks;       // chunks: packed chunks of K; split i works on [i * chunks / k_splits, (i + 1) * chunks / k_splits); k_splits = 1 << split_shift
    uint32_t raw_stages, stages, T;
    uint32_t early;              // packed weights may be fetched before the preceding kernel has finished
    uint32_t x_wrap;             // K after which the activation columns start over
    uint32_t M, N, K, layout, D;
    int* err;
    __half* Y;
    const __half* residual;
    float* scratch;              // [k_splits][tiles][T][128] partial tiles (k_splits > 1)
    const uint8_t* meta0;
    const __half* row_scale0;
    uint32_t n_tok_tiles;
    // SwiGLU and grouped launches
    uint32_t swiglu;             // tiles of 64 gate rows (matrix 0) and their 64 up rows (matrix 1); output silu(g) * u
    uint32_t groups, tiles[2];   // grouped launch: weight tiles [0, tiles[0]) belong to matrix 0, the next tiles[1] to matrix 1, ...
    uint32_t extra_N[2];         // features and results of the matrices behind the first
    __half* extra_Y[2];
    const uint8_t* meta1;
    const __half* row_scale1;
};
__device__ __forceinline__ float silu_mul(float g, float u) { return __fdividef(g, 1.0f + __expf(-g)) * u; }

__device__ __forceinline__ void tmem_st_x32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
          "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
          "r"(r[30]), "r"(r[31])
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]: fp16 operands, fp32 accumulate, A rows = tensor-memory lanes, K packed two per column
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ uint32_t cluster_ctarank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// words [W, HI) of a packed row; SW: the row was staged with the 128-byte TMA swizzle (16-byte chunk index ^ row % 8, the
// planar layouts' 128-byte rows) and is read in whole chunks
template <int W, int HI, bool SW = false>
__device__ __forceinline__ void ld_words(const uint8_t* rowp, uint32_t* r, uint32_t xr = 0u) {
    if constexpr (W < HI) {
        if constexpr (W % 4 == 0 && W + 4 <= HI) {
            const uint4 v = *reinterpret_cast<const uint4*>(rowp + (SW ? ((uint32_t)(W / 4) ^ xr) << 4 : (uint32_t)W * 4u));
            r[W] = v.x; r[W + 1] = v.y; r[W + 2] = v.z; r[W + 3] = v.w;
            ld_words<W + 4, HI, SW>(rowp, r, xr);
        } else if constexpr (W % 2 == 0 && W + 2 <= HI) {
            static_assert(!SW, "swizzled rows are read in 16-byte chunks");
            const uint2 v = *reinterpret_cast<const uint2*>(rowp + W * 4);
            r[W] = v.x; r[W + 1] = v.y;
            ld_words<W + 2, HI, SW>(rowp, r, xr);
        } else {
            static_assert(!SW, "swizzled rows are read in 16-byte chunks");
            r[W] = *reinterpret_cast<const uint32_t*>(rowp + W * 4);
            ld_words<W + 1, HI, SW>(rowp, r, xr);
        }
    }
}
template <int S> struct IntC { static constexpr int value = S; };
template <class F, int... S>
__device__ __forceinline__ void for_each_sub(F& f, std::integer_sequence<int, S...>) { (f(IntC<S>{}), ...); }

// Maps of the activations and of the packed matrices: one, or (MULTI: SwiGLU and grouped launches) up to three.  A plain launch has
// neither their maps among its parameters nor their branches.
template <bool MULTI> struct Maps { CUtensorMap x, w[MULTI ? 3 : 1]; };

template <int FMT, bool MULTI>
__global__ void __launch_bounds__(THREADS, 2)
qgemm_small_kernel(const __grid_constant__ Maps<MULTI> maps, const Params p) {
    const bool swiglu = MULTI && p.swiglu;
    using Cd = cdc::Codec<FMT>;
    constexpr int ROW_BYTES = Cd::ROW_BYTES;
    constexpr int RAW_TILE_BYTES = ROW_BYTES * W_TILE;
    constexpr int SUBS = Cd::CHUNK / KSTEP;
    constexpr bool SW = Cd::RAW_SWIZZLE_128;
    constexpr int MW = Cd::META_WORDS > 0 ? Cd::META_WORDS : 4;      // scale / bias words per chunk of the planar layouts

    extern __shared__ uint8_t smem_dyn[];
    ptx::launch_dependents();     // the next kernel in the stream may set itself up while this grid runs
    const uint32_t pad = (1024u - (ptx::smem_u32(smem_dyn) & 1023u)) & 1023u;
    uint8_t* sB = smem_dyn + pad;                                   // [B_STAGES][T rows of 128 bytes], 128-byte swizzle
    constexpr int SPS = Ring<FMT>::SPS, A_COLS = Ring<FMT>::A_COLS;
    const uint32_t b_sub_bytes = p.T * 128u, b_stage_bytes = SPS * b_sub_bytes;
    uint8_t* sRaw = sB + p.stages * b_stage_bytes;                  // [raw_stages][128 rows][ROW_BYTES]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sRaw + p.raw_stages * RAW_TILE_BYTES);
    uint64_t* raw_full = bars;
    uint64_t* raw_empty = raw_full + MAX_RAW_STAGES;
    uint64_t* full = raw_empty + MAX_RAW_STAGES;                    // step's weights in tensor memory (4 warps) and activations in shared memory
    uint64_t* empty = full + MAX_STAGES;                            // ... consumed: one tcgen05.commit
    uint64_t* acc_full = empty + MAX_STAGES;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_full + 1);
    volatile uint32_t* abort_flag = tmem_holder + 1;

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t ks = blockIdx.x & (p.k_splits - 1u);             // == rank inside the cluster
    const uint32_t tile = blockIdx.x >> p.split_shift;
    const uint32_t wt = tile % p.n_w_tiles, tt = tile / p.n_w_tiles;
    // grouped launch: this tile's matrix, and the tile's place in it
    uint32_t gi = 0u, wl = wt;
    if (MULTI && p.groups > 1u && wl >= p.tiles[0]) { wl -= p.tiles[0]; gi = 1u; if (wl >= p.tiles[1]) { wl -= p.tiles[1]; gi = 2u; } }
    const uint32_t N = !MULTI || gi == 0u ? p.N : (gi == 1u ? p.extra_N[0] : p.extra_N[1]);
    __half* const Y = !MULTI || gi == 0u ? p.Y : (gi == 1u ? p.extra_Y[0] : p.extra_Y[1]);
    const uint32_t kc0 = (ks * p.chunks) >> p.split_shift, kcn = (((ks + 1u) * p.chunks) >> p.split_shift) - kc0;     // this split's packed chunks
    const uint32_t ksteps = kcn * (uint32_t)(SUBS / SPS);

    if (threadIdx.x == 0) {
#pragma unroll
        for (uint32_t i = 0; i < (uint32_t)MAX_RAW_STAGES; i++) if (i < p.raw_stages) { ptx::mbar_init(&raw_full[i], 1); ptx::mbar_init(&raw_empty[i], UNPACK_WARPS); }
#pragma unroll
        for (uint32_t i = 0; i < (uint32_t)MAX_STAGES; i++) if (i < p.stages) { ptx::mbar_init(&full[i], UNPACK_WARPS + 1); ptx::mbar_init(&empty[i], 1); }
        ptx::mbar_init(acc_full, 1);
        *abort_flag = 0u;
        ptx::fence_barrier_init();
    }
    if (threadIdx.x == 0) QST(0, 0);
    if (warp == MMA_WARP) { ptx::tmem_alloc(tmem_holder, TMEM_COLS); ptx::tmem_relinquish(); }
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0) QST(0, 1);
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_holder;
    // Everything above touched only this CTA's shared and tensor memory.  Global memory is first touched below -- or, where the
    // preceding kernels are known not to write the weights, by the copies of packed chunks: they then stream in while the
    // preceding kernel drains, and the wait stands in front of the first activation tile and of the results.
    if (!p.early) ptx::grid_dependency_wait();
    if (threadIdx.x == 0) QST(0, 2);

    const uint32_t a_col = tmem_base + p.T;                         // A ring behind the accumulator
    if (warp == RAW_WARP) {
        // ---------------- packed weight chunks ----------------
        const CUtensorMap* tmW = &maps.w[MULTI ? gi : 0u];
        if (lane == 0) ptx::prefetch_tensormap(tmW);
        uint32_t rs = 0, rph = 0;
        bool ok = true;
        for (uint32_t kc = 0; kc < kcn; kc++) {
            ok = __all_sync(0xffffffffu, ptx::mbar_wait(&raw_empty[rs], rph ^ 1u, abort_flag, p.err, 111));
            if (!ok) break;
            if (lane == 0) {
                QST(1, kc);
                ptx::mbar_arrive_expect_tx(&raw_full[rs], RAW_TILE_BYTES);
                const int x = (int)((kc0 + kc) * (ROW_BYTES / Cd::TMA_ELEM_BYTES));
                if (swiglu) {          // 64-row boxes: gate rows, then the same rows of up
                    ptx::tma_load_2d(sRaw + rs * RAW_TILE_BYTES, &maps.w[0], &raw_full[rs], x, (int)(wt * GATE_ROWS));
                    ptx::tma_load_2d(sRaw + rs * RAW_TILE_BYTES + GATE_ROWS * ROW_BYTES, &maps.w[MULTI ? 1 : 0], &raw_full[rs], x, (int)(wt * GATE_ROWS));
                } else {
                    ptx::tma_load_2d(sRaw + rs * RAW_TILE_BYTES, tmW, &raw_full[rs], x, (int)(wl * W_TILE));
                }
            }
            __syncwarp();
            if (++rs == p.raw_stages) { rs = 0; rph ^= 1u; }
        }
    } else if (warp == ACT_WARP) {
        // ---------------- activation tiles ----------------
        if (lane == 0) ptx::prefetch_tensormap(&maps.x);
        if (p.early) ptx::grid_dependency_wait();
        uint32_t st = 0, ph = 0;
        bool ok = true;
        uint32_t x = (kc0 * (uint32_t)Cd::CHUNK) % p.x_wrap;      // column of the next activation tile (x_wrap: whole chunks)
        for (uint32_t k = 0; k < ksteps; k++) {
            ok = __all_sync(0xffffffffu, ptx::mbar_wait(&empty[st], ph ^ 1u, abort_flag, p.err, 112));
            if (!ok) break;
            if (lane == 0) {
                ptx::mbar_arrive_expect_tx(&full[st], b_stage_bytes);
                for (int j = 0; j < SPS; j++)
                    ptx::tma_load_2d(sB + st * b_stage_bytes + j * b_sub_bytes, &maps.x, &full[st], (int)x + j * KSTEP, (int)(tt * p.T));
            }
            __syncwarp();
            x += (uint32_t)(SPS * KSTEP);
            if (x == p.x_wrap) x = 0u;
            if (++st == p.stages) { st = 0; ph ^= 1u; }
        }
    } else if (warp == MMA_WARP) {
        // ---------------- MMA issuer: one thread, chosen once ----------------
        if (ptx::elect_one()) {
            const uint32_t idesc = ptx::umma_idesc_f16(W_TILE, p.T);
            const uint64_t desc_hi = ptx::umma_desc_k_sw128(0u);
            const uint32_t b_lo0 = (ptx::smem_u32(sB) & 0x3FFFFu) >> 4;
            uint32_t st = 0, ph = 0;
            for (uint32_t k = 0; k < ksteps; k++) {
                ptx::mbar_wait(&full[st], ph, abort_flag, p.err, 113);
                ptx::tc_fence_after_sync();
                QST(2, k);
                const uint64_t bdesc = desc_hi | (uint64_t)(b_lo0 + st * (b_stage_bytes >> 4));
                const uint32_t acol = a_col + st * A_COLS;
#pragma unroll
                for (int j = 0; j < SPS; j++)
#pragma unroll
                    for (int kk = 0; kk < KSTEP / 16; kk++)
                        umma_f16_ts(tmem_base, acol + j * SUB_COLS + kk * 8, bdesc + (uint64_t)(j * (b_sub_bytes >> 4) + 2 * kk), idesc, (k | (uint32_t)(j | kk)) != 0u);
                ptx::umma_commit(&empty[st]);
                if (++st == p.stages) { st = 0; ph ^= 1u; }
            }
            ptx::umma_commit(acc_full);
        }
        __syncwarp();
    } else {
        // ---------------- unpack: packed bytes -> registers -> tensor memory (A operand) ----------------
        const uint32_t quad = warp & 3u;                            // lane quadrant
        const uint32_t row = quad * 32u + lane;                     // weight row of the tile = tensor-memory lane
        const uint32_t lane_base = (quad * 32u) << 16;
        uint32_t rs = 0, rph = 0, st = 0, ph = 0;
        // (after a wait that gave up the rest runs out quickly, and nothing is written)
        for (uint32_t kc = 0; kc < kcn; kc++) {
            // planar layouts: this chunk's scales and biases come straight from their planes in global memory, requested
            // before the wait for the packed bytes
            uint32_t meta[MW] = {};
            if (Cd::META_WORDS != 0) {
                const uint32_t n = swiglu ? wt * GATE_ROWS + (row & 63u) : wt * W_TILE + row;
                if (n < p.N) {
                    const uint32_t groups = (p.K / 256u) * MW;
                    const uint8_t* mp = (swiglu && row >= 64u ? p.meta1 : p.meta0) + ((size_t)n * groups + (size_t)(kc0 + kc) * MW) * 2;
                    const uint8_t* bp = mp + (size_t)p.N * groups * 2;
                    if (MW == 4) {
                        const uint2 sc = ptx::ld(reinterpret_cast<const uint2*>(mp));
                        const uint2 bi = ptx::ld(reinterpret_cast<const uint2*>(bp));
                        meta[0] = sc.x; meta[1] = sc.y; meta[2] = bi.x; meta[3] = bi.y;
                    } else {
                        const uint4 sc = ptx::ld(reinterpret_cast<const uint4*>(mp));
                        const uint4 bi = ptx::ld(reinterpret_cast<const uint4*>(bp));
                        meta[0] = sc.x; meta[1] = sc.y; meta[2] = sc.z; meta[3] = sc.w;
                        meta[MW - 4] = bi.x; meta[MW - 3] = bi.y; meta[MW - 2] = bi.z; meta[MW - 1] = bi.w;
                    }
                }
            }
            ptx::mbar_wait(&raw_full[rs], rph, abort_flag, p.err, 115);
            if (threadIdx.x == 0) QST(3, kc);
            uint32_t r[ROW_BYTES / 4];
            const uint8_t* rowp = sRaw + rs * RAW_TILE_BYTES + row * ROW_BYTES;
            const uint32_t xr = row & 7u;
            ld_words<0, Cd::HDR_WORDS, SW>(rowp, r, xr);
            auto sub_tile = [&](auto S) {
                constexpr int s = decltype(S)::value;
                constexpr int j = s % SPS;                           // place inside the stage
                uint32_t o[32];
                ld_words<Cd::sub_lo(s), Cd::sub_hi(s), SW>(rowp, r, xr);
                Cd::dequant64(r, s, o, meta);
                if (j == 0) {
                    ptx::mbar_wait(&empty[st], ph ^ 1u, abort_flag, p.err, 116);
                    ptx::tc_fence_after_sync();                      // the MMAs that read this stage have completed
                }
                __syncwarp();                                        // (tensor memory is written by whole warps)
                tmem_st_x32(a_col + lane_base + st * A_COLS + j * SUB_COLS, o);
                if (j == SPS - 1) {
                    ptx::tmem_st_wait();
                    ptx::tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(&full[st]);
                    if (threadIdx.x == 0) QST(4, kc * SUBS + s);
                    if (++st == p.stages) { st = 0; ph ^= 1u; }
                }
            };
            for_each_sub(sub_tile, std::make_integer_sequence<int, SUBS>{});
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&raw_empty[rs]);         // after the stores that consumed every loaded register
            if (++rs == p.raw_stages) { rs = 0; rph ^= 1u; }
        }
    }

    // ---------------- partial tiles meet in the scratch buffer, the cluster shares out the sums ----------------
    if (p.early) ptx::grid_dependency_wait();      // (long over; orders this thread's stores behind it)
    if (warp < 4) {
        // the accumulator is complete once every MMA has; a failed wait sets the abort flag, the barrier is still reached
        ptx::mbar_wait(acc_full, 0u, abort_flag, p.err, 117);
    }
    __syncthreads();
    if (threadIdx.x == 0) QST(0, 3);
    const bool bad = *abort_flag != 0u;
    const uint32_t n_tiles = p.n_w_tiles * p.n_tok_tiles;
    const size_t tile_floats = (size_t)p.T * W_TILE;
    if (warp < 4 && !bad) {
        ptx::tc_fence_after_sync();
        const uint32_t f = warp * 32u + lane;                       // feature row of the tile
        const uint32_t n = swiglu ? wt * GATE_ROWS + (f & 63u) : wl * W_TILE + f;
        float rsc = 1.0f;
        if (Cd::ROW_SCALE) rsc = n < N ? __half2float((swiglu && f >= 64u ? p.row_scale1 : p.row_scale0)[n]) : 0.0f;
        const uint32_t taddr = tmem_base + ((warp * 32u) << 16);
        if (swiglu && p.k_splits == 1u) {
            // A whole SwiGLU tile: lanes 0 .. 63 hold the gate projections of 64 features, lanes 64 .. 127 the up projections of the same.
            // 16 token columns at a time change hands through the operand rings, which nothing reads any more, and leave as whole rows
            // of the tile (F = 14336, K = 4096, 128 tokens 32.1 us; through the scratch buffer and back, like split sums, 39.0).
            float* stage = reinterpret_cast<float*>(sB);                 // [2][16 columns][128 features]
            const uint32_t tok0 = tt * p.T, valid = min(p.T, p.M - tok0), col = threadIdx.x >> 3, f0 = (threadIdx.x & 7u) * 8u, n0 = wt * GATE_ROWS + f0;
            const bool wide = N % 8u == 0u && (reinterpret_cast<uintptr_t>(Y) & 15u) == 0;
            for (uint32_t c0 = 0, b = 0; c0 < valid; c0 += 16u, b ^= 1u) {
                uint32_t v[16];
                __syncwarp();                                            // (tensor memory is read by whole warps)
                ptx::tmem_ld_x16(taddr + c0, v);
                ptx::tmem_ld_wait();
                float* buf = stage + b * (16 * W_TILE);
#pragma unroll
                for (int j = 0; j < 16; j++) buf[j * W_TILE + f] = Cd::ROW_SCALE ? __uint_as_float(v[j]) * rsc : __uint_as_float(v[j]);
                ptx::bar_sync(1, 128);                                   // (the buffer after next is written behind the next barrier)
                if (c0 + col >= valid) continue;
                const float4* g = reinterpret_cast<const float4*>(buf + col * W_TILE + f0);
                const float4 g0 = g[0], g1 = g[1], u0 = g[GATE_ROWS / 4], u1 = g[GATE_ROWS / 4 + 1];
                const float a[8] = {silu_mul(g0.x, u0.x), silu_mul(g0.y, u0.y), silu_mul(g0.z, u0.z), silu_mul(g0.w, u0.w),
                                    silu_mul(g1.x, u1.x), silu_mul(g1.y, u1.y), silu_mul(g1.z, u1.z), silu_mul(g1.w, u1.w)};
                __half* dst = Y + (size_t)(tok0 + c0 + col) * N + n0;
                if (wide && n0 < N) {
                    __half2 h[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) h[e] = __floats2half2_rn(a[2 * e], a[2 * e + 1]);
                    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(h);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; e++) if (n0 + e < N) dst[e] = __float2half_rn(a[e]);
                }
            }
        } else if (p.k_splits > 1u) {
            // [split][tile][token column][feature]: a warp's store covers 32 consecutive features of one column
            float* dst = p.scratch + ((size_t)ks * n_tiles + tile) * tile_floats + f;
            const uint32_t valid = min(p.T, p.M - tt * p.T);
            for (uint32_t c0 = 0; c0 < valid; c0 += 16) {
                uint32_t v[16];
                ptx::tmem_ld_x16(taddr + c0, v);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (c0 + j < valid) __stcg(dst + (size_t)(c0 + j) * W_TILE, Cd::ROW_SCALE ? __uint_as_float(v[j]) * rsc : __uint_as_float(v[j]));
            }
        } else {
            // no split: this CTA's accumulator is the result
            const uint32_t tok0 = tt * p.T;
            for (uint32_t c0 = 0; c0 < p.T; c0 += 16) {
                uint32_t v[16];
                ptx::tmem_ld_x16(taddr + c0, v);
                ptx::tmem_ld_wait();
                if (n >= N) continue;
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const uint32_t tok = tok0 + c0 + j;
                    if (tok >= p.M) break;
                    float a = Cd::ROW_SCALE ? __uint_as_float(v[j]) * rsc : __uint_as_float(v[j]);
                    const size_t o = p.layout == 1 ? ((size_t)(n / p.D) * p.M + tok) * p.D + (n % p.D) : (size_t)tok * N + n;
                    if (p.residual) a += __half2float(p.residual[o]);
                    Y[o] = __float2half_rn(a);
                }
            }
        }
    }
    if (threadIdx.x == 0) QST(0, 5);
    // every partial tile of the cluster is written (release / acquire at cluster scope covers the global stores)
    cluster_sync_all();
    if (threadIdx.x == 0) QST(0, 6);
    if (!bad && p.k_splits > 1u) {
        // this CTA's token columns [ks * cols, (ks + 1) * cols): sum over the splits in split order, write fp16
        const uint32_t cols = p.T >> p.split_shift;
        const float* base = p.scratch + (size_t)tile * tile_floats + (size_t)(ks * cols) * W_TILE;
        const size_t split_stride = (size_t)n_tiles * tile_floats;
        const uint32_t tok0 = tt * p.T + ks * cols;
        // two float4 of every split at a time -- items i and i + THREADS, or (SwiGLU) the gate and the up value of one item -- four
        // splits' loads under way together
        auto sum4x2 = [&](const float* a, const float* b, bool both, float4& x, float4& y) {
            x = y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (uint32_t s0 = 0; s0 < p.k_splits; s0 += 4u) {
                float4 v[4], w[4];
#pragma unroll
                for (uint32_t j = 0; j < 4u; j++) {
                    const size_t o = (s0 + j) * split_stride;
                    v[j] = w[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (s0 + j < p.k_splits) v[j] = __ldcg(reinterpret_cast<const float4*>(a + o));
                    if (s0 + j < p.k_splits && both) w[j] = __ldcg(reinterpret_cast<const float4*>(b + o));
                }
#pragma unroll
                for (uint32_t j = 0; j < 4u; j++) {
                    x.x += v[j].x; x.y += v[j].y; x.z += v[j].z; x.w += v[j].w;
                    y.x += w[j].x; y.y += w[j].y; y.z += w[j].z; y.w += w[j].w;
                }
            }
        };
        // four features per item; a SwiGLU tile's features 64 .. 127 are the up projections of 0 .. 63
        const uint32_t quads = swiglu ? GATE_ROWS / 4 : W_TILE / 4, quad_shift = swiglu ? 4u : 5u;
        const uint32_t valid = tok0 < p.M ? min(cols, p.M - tok0) : 0u, items = valid << quad_shift;
        static_assert(GATE_ROWS == 64 && W_TILE == 128, "quads per column: 16 and 32");
        auto write4 = [&](uint32_t i, float4 acc) {
            const uint32_t f = (i & (quads - 1u)) * 4u, tok = tok0 + (i >> quad_shift), n = swiglu ? wt * GATE_ROWS + f : wl * W_TILE + f;
            const float a[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (n + e >= N) break;
                const size_t o = p.layout == 1 ? ((size_t)((n + e) / p.D) * p.M + tok) * p.D + ((n + e) % p.D) : (size_t)tok * N + n + e;
                Y[o] = __float2half_rn(p.residual ? a[e] + __half2float(p.residual[o]) : a[e]);
            }
        };
        for (uint32_t i = threadIdx.x; i < items; i += swiglu ? THREADS : 2 * THREADS) {
            const uint32_t i2 = i + THREADS;
            const float* at = base + (size_t)(i >> quad_shift) * W_TILE + (i & (quads - 1u)) * 4u;
            const float* at2 = swiglu ? at + GATE_ROWS : base + (size_t)(i2 >> quad_shift) * W_TILE + (i2 & (quads - 1u)) * 4u;
            float4 x, y;
            sum4x2(at, at2, swiglu || i2 < items, x, y);
            if (swiglu) write4(i, make_float4(silu_mul(x.x, y.x), silu_mul(x.y, y.y), silu_mul(x.z, y.z), silu_mul(x.w, y.w)));
            else { write4(i, x); if (i2 < items) write4(i2, y); }
        }
    }
    // ---------------- teardown ----------------
    if (threadIdx.x == 0) QST(0, 7);
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (bad) {      // let copies that are still in flight land before the CTA gives its shared memory back
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000LL) { }
        __syncthreads();
    }
    if (warp == MMA_WARP) { ptx::tc_fence_after_sync(); ptx::tmem_dealloc(tmem_base, TMEM_COLS); }
    if (threadIdx.x == 0) QST(0, 8);
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
bool make_map(CUtensorMap* m, CUtensorMapDataType dt, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_bytes,
              uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle sw) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {row_bytes};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t estr[2] = {1, 1};
    return fn(m, dt, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct Plan { uint32_t T, n_tok_tiles, n_w_tiles, k_splits, chunks, raw_stages, stages; size_t smem; };

// alignment slack + activation ring + packed ring + barrier block
template <int FMT> size_t smem_bytes(uint32_t T, uint32_t raw_stages, uint32_t stages) {
    return 1024 + (size_t)stages * T * 128 * Ring<FMT>::SPS + (size_t)raw_stages * cdc::Codec<FMT>::ROW_BYTES * W_TILE + 256;
}
// Operand stages: as many as tensor memory holds behind the accumulator
template <int FMT> void stages_for(uint32_t T, uint32_t chunks, uint32_t& raw, uint32_t& stages) {
    stages = (TMEM_COLS - T) / Ring<FMT>::A_COLS;
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    while (stages > 2u && smem_bytes<FMT>(T, 2, stages) > SMEM_LIMIT) stages--;          // (the 272-byte rows at 128 tokens: two)
    raw = 2;
    while (raw < (uint32_t)MAX_RAW_STAGES && raw < chunks && smem_bytes<FMT>(T, raw + 1, stages) <= SMEM_LIMIT) raw++;
}

int g_sms = 0;
int sms() {
    if (!g_sms) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev); if (g_sms <= 0) g_sms = 148; }
    return g_sms;
}

template <int FMT> bool make_plan(const GemmArgs& a, Plan& pl) {
    using Cd = cdc::Codec<FMT>;
    static_assert(1024 + 2 * MAX_T * 128 * Ring<FMT>::SPS + 2 * Cd::ROW_BYTES * W_TILE + 256 <= SMEM_LIMIT, "two stages of each ring fit half an SM");
    pl.n_tok_tiles = (a.M + MAX_T - 1) / MAX_T;
    const uint32_t per = (a.M + pl.n_tok_tiles - 1) / pl.n_tok_tiles;
    pl.T = (per + 15u) & ~15u;
    const uint32_t rows_per_tile = a.W1 ? GATE_ROWS : W_TILE;        // output features per tile
    pl.n_w_tiles = (a.N + rows_per_tile - 1) / rows_per_tile;
    for (uint32_t e = 0; e < a.n_extra && e < 2u; e++) pl.n_w_tiles += (a.N_extra[e] + W_TILE - 1) / W_TILE;
    const uint32_t chunks = a.K / Cd::CHUNK;
    const uint32_t tiles = pl.n_tok_tiles * pl.n_w_tiles;
    // split K while all CTAs still fit on the GPU at two per SM, every split keeps a whole chunk, and the token columns
    // divide evenly among the CTAs of a cluster
    pl.k_splits = 1;
    for (uint32_t s = 2; s <= 8; s *= 2) {
        if (tiles * s > 2u * (uint32_t)sms() || chunks < s || pl.T % s != 0) break;
        if (a.lean && chunks % s != 0) break;
        if (a.n_extra && chunks / s < 2) break;       // grouped launches: the persistent kernel's rule, so that both split alike
        pl.k_splits = s;
    }
    pl.chunks = chunks;
    // at least 80 KB, so that no more than two CTAs share an SM: each holds 256 of the SM's 512 tensor-memory columns, and a
    // third CTA would sit in tcgen05.alloc until one of the others leaves
    stages_for<FMT>(pl.T, (chunks + pl.k_splits - 1) / pl.k_splits, pl.raw_stages, pl.stages);
    pl.smem = smem_bytes<FMT>(pl.T, pl.raw_stages, pl.stages);
    if (pl.smem < 80 * 1024) pl.smem = 80 * 1024;
    return tiles * pl.k_splits <= 65535u * 8u;
}

template <int FMT> size_t scratch_floats_fmt(const GemmArgs& a) {
    Plan pl;
    if (!make_plan<FMT>(a, pl) || pl.k_splits <= 1) return 0;
    return (size_t)pl.k_splits * pl.n_tok_tiles * pl.n_w_tiles * pl.T * W_TILE;
}

template <int FMT, bool MULTI> cudaError_t launch_multi(const GemmArgs& a, const Workspace& ws, cudaStream_t stream) {
    using Cd = cdc::Codec<FMT>;
    Plan pl;
    if (!make_plan<FMT>(a, pl)) return cudaErrorInvalidValue;
    if (pl.k_splits > 1 && (!ws.partial || ws.partial_floats < (size_t)pl.k_splits * pl.n_tok_tiles * pl.n_w_tiles * pl.T * W_TILE))
        return cudaErrorInvalidValue;
    const uint64_t w_row_bytes = (uint64_t)(a.K / Cd::CHUNK) * Cd::ROW_BYTES;
    const uint32_t x_cols = a.x_cols ? a.x_cols : a.K;          // columns past the end read as zero
    Maps<MULTI> maps;
    if (!make_map(&maps.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.X, x_cols, a.M, (uint64_t)x_cols * 2, KSTEP, pl.T, CU_TENSOR_MAP_SWIZZLE_128B))
        return cudaErrorInvalidValue;
    constexpr int EB = Cd::TMA_ELEM_BYTES;
    auto weight_map = [&](CUtensorMap* m, const void* w, uint32_t n) {
        return make_map(m, EB == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, w, w_row_bytes / EB, n, w_row_bytes,
                        Cd::ROW_BYTES / EB, a.W1 ? GATE_ROWS : W_TILE, Cd::RAW_SWIZZLE_128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE);
    };
    // second and third map: the up matrix of a SwiGLU launch, or the extra matrices of a grouped one
    if (!weight_map(&maps.w[0], a.W0, a.N)) return cudaErrorInvalidValue;
    if constexpr (MULTI) {
        maps.w[1] = maps.w[2] = maps.w[0];
        if (a.W1 && !weight_map(&maps.w[1], a.W1, a.N)) return cudaErrorInvalidValue;
        for (uint32_t e = 0; e < a.n_extra; e++)
            if (!weight_map(&maps.w[1 + e], a.W_extra[e], a.N_extra[e])) return cudaErrorInvalidValue;
    }
    Params p;
    p.M = a.M; p.N = a.N; p.K = a.K; p.T = pl.T; p.x_wrap = a.x_wrap ? a.x_wrap : a.K;
    p.n_tok_tiles = pl.n_tok_tiles; p.n_w_tiles = pl.n_w_tiles; p.k_splits = pl.k_splits; p.chunks = pl.chunks;
    p.split_shift = 0u;
    while ((1u << p.split_shift) < pl.k_splits) p.split_shift++;
    p.raw_stages = pl.raw_stages; p.stages = pl.stages; p.early = a.early_weights ? 1u : 0u; p.swiglu = a.W1 ? 1u : 0u;
    p.groups = 1u + a.n_extra;
    p.Y = (__half*)a.Y;
    p.tiles[0] = (a.N + W_TILE - 1) / W_TILE; p.tiles[1] = a.n_extra ? (a.N_extra[0] + W_TILE - 1) / W_TILE : 0u;
    for (uint32_t e = 0; e < 2u; e++) { p.extra_N[e] = e < a.n_extra ? a.N_extra[e] : 0u; p.extra_Y[e] = e < a.n_extra ? (__half*)a.Y_extra[e] : nullptr; }
    p.residual = (const __half*)a.residual; p.layout = (uint32_t)a.layout; p.D = a.D ? a.D : 2;
    p.err = ws.err; p.scratch = ws.partial;
    p.meta0 = (const uint8_t*)a.W0 + (size_t)a.N * w_row_bytes;
    p.meta1 = a.W1 ? (const uint8_t*)a.W1 + (size_t)a.N * w_row_bytes : p.meta0;
    p.row_scale0 = (const __half*)p.meta0; p.row_scale1 = (const __half*)p.meta1;
    static uint64_t attr_mask = 0;
    static std::mutex mu;
    {
        int dev = 0;
        cudaGetDevice(&dev);
        std::lock_guard<std::mutex> lock(mu);
        if (!(dev >= 0 && dev < 64 && ((attr_mask >> dev) & 1u))) {
            cudaError_t e = cudaFuncSetAttribute(qgemm_small_kernel<FMT, MULTI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_LIMIT);
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) attr_mask |= 1ull << dev;
        }
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(pl.n_tok_tiles * pl.n_w_tiles * pl.k_splits);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = pl.k_splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // prologue may overlap the previous kernel's tail
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, qgemm_small_kernel<FMT, MULTI>, maps, p);
}

template <int FMT> cudaError_t launch_fmt(const GemmArgs& a, const Workspace& ws, cudaStream_t stream) {
    return a.W1 || a.n_extra ? launch_multi<FMT, true>(a, ws, stream) : launch_multi<FMT, false>(a, ws, stream);
}

int g_mode = 1;

}  // namespace
}  // namespace small

void set_small_kernel_enabled(int mode) { small::g_mode = mode; }

#ifdef QS_TRACE
extern "C" int b200_debug_small_trace(unsigned long long* out) {
    return cudaMemcpyFromSymbol(out, small::g_qs_trace, sizeof(small::g_qs_trace)) == cudaSuccess ? 0 : -1;
}
#endif

bool small_path_ok(const GemmArgs& a) {
    if (small::g_mode == 0 || a.force_generic) return false;
    if (a.partial_out || a.scatter.world || a.wait_rows.flags || a.post[0] || a.post[1] || a.post[2]) return false;
    if (a.lean && (a.W1 || a.n_extra || (a.N + 127u) / 128u >= (uint32_t)small::sms())) return false;
    if (a.W1 && (((uintptr_t)a.W1 & 15u) || a.residual || a.layout != 0 || a.n_extra)) return false;
    // (matrices of a grouped launch: plain block formats, as on the persistent kernel)
    if (a.n_extra && (a.n_extra > 2 || a.residual || a.format == QUANT_TERNARY_ROW || a.format == QUANT_MLX_4BIT_G64 || a.format == QUANT_MLX_4BIT_PLANAR)) return false;
    for (uint32_t e = 0; e < a.n_extra && e < 2u; e++)
        if (!a.W_extra[e] || ((uintptr_t)a.W_extra[e] & 15u) || !a.Y_extra[e] || a.N_extra[e] == 0) return false;
    if (a.M == 0 || a.N == 0 || a.K == 0) return false;
    if (((uintptr_t)a.X & 15u) || ((uintptr_t)a.W0 & 15u) || ((uintptr_t)a.Y & 3u)) return false;
    if (a.residual && (a.layout != 0 || ((uintptr_t)a.residual & 1u))) return false;
    if (a.layout == 1 && (a.D == 0 || a.D % 2u != 0u)) return false;
    uint32_t chunk = 256;
    switch (a.format) {
        case QUANT_Q4_0: case QUANT_MLX_4BIT: case QUANT_Q4_K: case QUANT_TERNARY_1_58: case QUANT_VAR_RATE_AFFINE: case QUANT_EXL3:
        case QUANT_TERNARY_ROW: case QUANT_MLX_4BIT_G64: case QUANT_MLX_4BIT_PLANAR: break;
        case QUANT_PRISM_Q2_0: chunk = 1024; break;
        default: return false;
    }
    if (a.K % chunk != 0) return false;
    if (small::g_mode == 2) return true;
    // More than one token tile unpacks every weight tile more than once, which costs nothing where most of the GPU would idle: where
    // the persistent kernel (an SM per CTA) has so few tiles that it could split a long K eight ways, this one has its work in twice
    // as many CTAs (160 tokens, K = 4096, N = 2048 19.3 -> 12.3 us).  Its clusters of eight have to be resident at once: 32 of them
    // are, 36 are not (an eighth of the SMs is left over where a GPC is not whole clusters).  Below 16 tiles the persistent kernel
    // is as fast; in the variable-rate format unpacking twice does cost (1.2 to 1.4 times).
    if (a.M > (uint32_t)small::MAX_T) {
        if (a.W1 || a.n_extra || a.lean || a.format == QUANT_VAR_RATE_AFFINE || a.K / chunk < 16u) return false;
        const uint32_t w_tiles = (a.N + 127u) / 128u, tiles = (a.M + 127u) / 128u * w_tiles, persistent = (a.M + 255u) / 256u * w_tiles;
        return tiles >= 16u && persistent * 8u <= (uint32_t)small::sms() && tiles * 8u <= (uint32_t)small::sms() / 4u * 7u;
    }
    // One token tile: at most two weight tiles per SM.  Beyond that the persistent kernel, which starts on the next tile while the
    // last one drains, is as fast.
    uint32_t tiles = a.W1 ? (a.N + small::GATE_ROWS - 1) / small::GATE_ROWS : (a.N + 127u) / 128u;
    for (uint32_t e = 0; e < a.n_extra && e < 2u; e++) tiles += (a.N_extra[e] + 127u) / 128u;
    if (tiles > 2u * (uint32_t)small::sms()) return false;
    // With more SwiGLU tiles than SMs K is not split, and the tiles leave straight from the accumulator: always better here (F = 14336,
    // K = 4096: 33 tokens 27.0 us, 41.1 on the persistent kernel; 128 tokens 31.8, 44.5).  Fewer tiles are split (K of one chunk
    // apart) and pass through the scratch buffer, which grows with the tokens: a short K does not make up for it (F = 5632: K = 512,
    // 64 tokens 8.3 against 7.3 us; K = 1024, 64 tokens 9.4 against 9.8), in the variable-rate format a shorter one does.
    const uint32_t T = (a.M + 15u) & ~15u;
    // Grouped launches with a short K for their tokens: the same (1024 + 2 x 256 features, K = 1024: 64 tokens 10.4 against 10.8 us,
    // 128 tokens 14.3 against 12.5), and earlier in the variable-rate format (K = 512, one token 9.3 against 7.6).
    if (a.n_extra && (a.format == QUANT_VAR_RATE_AFFINE ? a.K <= 512u || a.K < 22u * T : a.K < 12u * T)) return false;
    if (a.W1 && tiles <= (uint32_t)small::sms() && a.K < (a.format == QUANT_VAR_RATE_AFFINE ? 8u : 10u) * T) return false;
    return true;
}

#define QG_SMALL_DISPATCH(EXPR)                                                            \
    switch (a.format) {                                                                    \
        case QUANT_Q4_0: { constexpr int F = QUANT_Q4_0; return EXPR; }                    \
        case QUANT_MLX_4BIT: { constexpr int F = QUANT_MLX_4BIT; return EXPR; }            \
        case QUANT_Q4_K: { constexpr int F = QUANT_Q4_K; return EXPR; }                    \
        case QUANT_TERNARY_1_58: { constexpr int F = QUANT_TERNARY_1_58; return EXPR; }    \
        case QUANT_VAR_RATE_AFFINE: { constexpr int F = QUANT_VAR_RATE_AFFINE; return EXPR; } \
        case QUANT_EXL3: { constexpr int F = QUANT_EXL3; return EXPR; }                    \
        case QUANT_TERNARY_ROW: { constexpr int F = QUANT_TERNARY_ROW; return EXPR; }      \
        case QUANT_MLX_4BIT_G64: { constexpr int F = QUANT_MLX_4BIT_G64; return EXPR; }    \
        case QUANT_MLX_4BIT_PLANAR: { constexpr int F = QUANT_MLX_4BIT_PLANAR; return EXPR; } \
        case QUANT_PRISM_Q2_0: { constexpr int F = QUANT_PRISM_Q2_0; return EXPR; }        \
        default: break;                                                                    \
    }

cudaError_t launch_small(const GemmArgs& a, const Workspace& ws, cudaStream_t stream) {
    QG_SMALL_DISPATCH(small::launch_fmt<F>(a, ws, stream))
    return cudaErrorInvalidValue;
}

size_t small_scratch_floats(const GemmArgs& a) {
    QG_SMALL_DISPATCH(small::scratch_floats_fmt<F>(a))
    return 0;
}

}  // namespace qg
