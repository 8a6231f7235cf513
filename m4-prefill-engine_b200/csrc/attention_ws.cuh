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
cudaError_t launch(const Args& a, cudaStream_t stream, int* launches);

}  // namespace ws
}  // namespace attn
