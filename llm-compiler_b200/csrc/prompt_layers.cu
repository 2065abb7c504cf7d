// The layers of a Qwen2 prompt, launched from one call. A short prompt is some eight launches a layer of 2 - 14 us each;
// issued one by one from Python (checks, output tensors, argument conversion: 13 us a launch, of which the launch
// itself is 4) the GPU waited for the host. Qwen2-0.5B, 77 tokens: 5.1 ms of host work for 1.8 ms of kernels.
#include "common.cuh"
#include "prompt_layers.cuh"

using namespace b200;

extern "C" int b200_qwen2_prompt_layers(const b200_prompt_layer* layers, int64_t num_layers,
                                        const b200_prompt_call* c, int32_t* status, void* stream) {
  if (!layers || !c || num_layers < 0 || !c->x || !c->x_middle || !c->h || !c->qkv || !c->q || !c->k || !c->attention ||
      !c->gated || !c->cosine || !c->sine || !c->positions || c->batch < 0 || c->tokens < 0 || c->q_heads <= 0 ||
      c->kv_heads <= 0 || c->head_dim <= 0 || c->hidden <= 0 || c->intermediate <= 0 || c->capacity < c->tokens)
    return B200_ERR_BAD_ARGUMENT;
  if (!known_dtype(c->dtype)) return B200_ERR_UNSUPPORTED;
  const int64_t batch = c->batch, tokens = c->tokens, rows = batch * tokens, dim = c->head_dim;
  if (rows == 0) return B200_OK;
  const int64_t q_size = c->q_heads * dim, kv_size = c->kv_heads * dim, width = q_size + 2 * kv_size;
  const size_t size = dtype_bytes(c->dtype);
  const char* qkv = static_cast<const char*>(c->qkv);
  const void *q_in = qkv, *k_in = qkv + q_size * size, *v_in = qkv + (q_size + kv_size) * size;
  const int64_t packed[4] = {tokens * width, dim, width, 1};           // a part of the projection as B, H, T, D
  const int64_t table[3] = {tokens * dim, dim, 1};
  const int64_t q_strides[4] = {tokens * q_size, tokens * dim, dim, 1};   // rotated: B, H, T, D
  const int64_t k_strides[4] = {tokens * kv_size, tokens * dim, dim, 1};
  const int64_t cached[4] = {c->capacity * kv_size, dim, kv_size, 1};  // a buffer as B, H, T, D
  for (int64_t i = 0; i < num_layers; ++i) {
    const b200_prompt_layer& l = layers[i];
    auto norm = [&](const void* x, const void* weight) {
      return b200_rms_norm(x, weight, c->h, rows, c->hidden, c->hidden, c->epsilon, 1, c->dtype, c->dtype, c->dtype,
                           c->mode, stream);
    };
    auto linear = [&](const void* x, const void* weight, const void* bias, const void* residual, void* out, int64_t k,
                      int64_t n, int epilogue) {
      return b200_linear(x, weight, bias, residual, out, rows, k, n, k, c->dtype, epilogue, c->workspace,
                         c->workspace_bytes, status, stream);
    };
    int code = norm(c->x, l.input_norm);
    if (code == B200_OK)
      code = linear(c->h, l.qkv_weight, l.qkv_bias, nullptr, c->qkv, c->hidden, width, B200_EPILOGUE_NONE);
    if (code != B200_OK) return code;
    const void *keys = c->k, *values = v_in;
    const int64_t *key_strides = k_strides, *value_strides = packed;
    code = c->block_table != nullptr
               ? B200_ERR_UNSUPPORTED
               : rope_into_cache(c->qkv, c->cosine, c->sine, c->q, l.keys, l.values, batch, tokens, c->q_heads,
                                 c->kv_heads, dim, c->capacity, c->dtype, static_cast<cudaStream_t>(stream));
    if (code == B200_OK) {  // attention reads what was stored
      keys = l.keys;
      values = l.values;
      key_strides = value_strides = cached;
    } else if (code == B200_ERR_UNSUPPORTED) {  // a block pool, or rows without 16-byte access
      code = b200_rope(q_in, k_in, c->cosine, c->sine, c->q, c->k, batch, c->q_heads, c->kv_heads, tokens, dim, packed,
                       packed, table, table, c->dtype, stream);
      if (code == B200_OK && c->block_table != nullptr)
        code = b200_paged_kv_store(l.keys, l.values, c->block_table, c->k, v_in, c->positions, batch, c->kv_heads, tokens,
                                   dim, c->num_blocks, c->block_size, c->max_blocks, k_strides, packed, c->dtype, status,
                                   stream);
      else if (code == B200_OK)
        code = b200_kv_store(l.keys, l.values, c->k, v_in, c->positions, batch, c->capacity, c->kv_heads, tokens, dim,
                             k_strides, packed, c->dtype, status, stream);
    }
    if (code == B200_OK)
      code = b200_prefill_attention(c->q, keys, values, nullptr, c->attention, batch, c->q_heads, c->kv_heads, tokens, dim,
                                    q_strides, key_strides, value_strides, nullptr, B200_F32, c->scale, 1, c->dtype,
                                    c->mode, nullptr, 0, status, stream);
    if (code == B200_OK)
      code = linear(c->attention, l.o_weight, nullptr, c->x, c->x_middle, q_size, c->hidden, B200_EPILOGUE_RESIDUAL);
    if (code == B200_OK) code = norm(c->x_middle, l.post_norm);
    if (code == B200_OK)
      code = linear(c->h, l.gate_up_weight, nullptr, nullptr, c->gated, c->hidden, 2 * c->intermediate,
                    B200_EPILOGUE_SWIGLU);
    if (code == B200_OK)
      code = linear(c->gated, l.down_weight, nullptr, c->x_middle, c->x, c->intermediate, c->hidden,
                    B200_EPILOGUE_RESIDUAL);
    if (code != B200_OK) return code;
  }
  return B200_OK;
}
