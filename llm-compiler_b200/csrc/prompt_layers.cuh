#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

// RoPE and KV store of a prompt from position 0 on, in one pass over the stacked projection qkv [batch, tokens, q | k | v]:
// rotated q as B, H, T, D into q_out, rotated k and v into the buffers [batch, capacity, kv_heads, head_dim]. cosine /
// sine: [batch, tokens, head_dim]. B200_ERR_UNSUPPORTED where the rows do not allow 16-byte accesses.
int rope_into_cache(const void* qkv, const void* cosine, const void* sine, void* q_out, void* keys, void* values,
                    int64_t batch, int64_t tokens, int64_t q_heads, int64_t kv_heads, int64_t head_dim, int64_t capacity,
                    int dtype, cudaStream_t stream);

}  // namespace b200
