// Host-side interface of the tensor-memory attention kernel (attention_ws.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace attn {
namespace ws {

struct Args {
    const void *Q, *K, *V;       // device; K and V as Q8_0 records, or fp16 when kv_fp16
    void* O;
    uint32_t Hq, Hkv, M, Mkv, D, pos0;
    float scale_log2e;
    int out_tokens_major, kv_fp16;
};

// head dim 64 or 128, at most 128 query heads per kv head, 16-byte-aligned Q and O (and K, V when fp16), positive scale
bool usable(const Args& a);
// How a launch is cut up: query tiles of a CTA and position blocks, splits of the key range (one, unless `split`), keys that some
// row sees, and the scratch that takes: the expanded Q8_0 cache, then the partial results of the splits.
struct Plan {
    uint32_t BP, tiles, blocks, n_last, splits, kv_rows;
    size_t kv_bytes, o_bytes, ml_bytes;
    size_t scratch_bytes() const { return kv_bytes + o_bytes + ml_bytes; }
};
Plan make_plan(const Args& a, bool split);
// The scratch is the caller's for as long as the launch may run (a captured launch: as long as its graph lives).  With less than
// the plan asks for the key range stays whole; with less than make_plan(a, false) does, the answer is cudaErrorMemoryAllocation.
struct Scratch { void* p; size_t bytes; };
cudaError_t launch(const Args& a, const Plan& plan, const Scratch& scratch, cudaStream_t stream, int* launches);

}  // namespace ws
}  // namespace attn
