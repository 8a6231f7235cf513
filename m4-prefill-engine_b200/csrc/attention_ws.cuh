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
// Scratch of a launch, the caller's for as long as the launch may run (a captured launch: as long as its graph lives): the expanded
// Q8_0 cache, then the partial results of a split key range.  With less than scratch_bytes(a, true) the key range stays whole,
// with less than scratch_bytes(a, false) launch() answers cudaErrorMemoryAllocation.
struct Scratch { void* p; size_t bytes; };
size_t scratch_bytes(const Args& a, bool split);
cudaError_t launch(const Args& a, const Scratch& scratch, cudaStream_t stream, int* launches);

}  // namespace ws
}  // namespace attn
