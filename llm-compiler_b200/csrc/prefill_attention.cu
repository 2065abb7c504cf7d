// serve.prefill_attention: T-token GQA attention with an arbitrary additive
// B x 1 x T x T mask, or with proven causality (fully masked key tiles are skipped and
// the mask is not read).
//
// bf16 / fp16 kernel (warp-level tensor cores): a CTA of 4 warps owns 64 query rows of one
// (sequence, q head); each warp keeps 16 rows of Q as A fragments and streams 64-key
// K/V tiles through a cp.async ring of XOR-swizzled rows; S = Q K^T and O += P V are
// m16n8k16 tiles with an fp32 online softmax in the log2 domain. The output is written
// token-major (B x T x Hq x D) so that the transpose + reshape that follows in the
// graph is a view.
//
// fp16 takes this kernel for every mask and mode. Its scores stay in the natural domain (an additive mask may hold
// the type's lowest value, whose multiple by log2 e would overflow to -inf and turn a uniform row into NaN), and
// its probabilities stay fp32 numbers: expf as in the CUDA-core kernel, and 2^15 p enters P V as three fp16 operands with
// sums of their own, 2^15 p rounded, then 2^11 times what is left, twice: 33 bits, and no probability above 2^-62 of the
// row's largest is lost (as one fp16 number those below 2^-25 would count in the denominator only). The sums of a key
// tile are added to the running output in fp32: tensor cores cut an accumulator's last bits off at every step, and a
// chain through the whole context would show it. Errors against 64 bits at 130 - 4096 tokens are those of the CUDA-core
// kernel to four digits. 2 x 515 tokens, 14 heads of 64: 1851 us on the CUDA-core kernel (one CTA per
// query row, keys and values re-read by every row) -> 36 us (26 with one remainder and a chain through the context).
//
// fp32 kernel: CUDA cores with IEEE fp32 dots for small full-precision graphs.
#include <math.h>

#include "common.cuh"

namespace b200 {
namespace {

constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kBM = 64;  // query rows per CTA
constexpr int kBN = 64;  // keys per tile
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kHalfScale = 32768.0f, kPartScale = 2048.0f;  // of fp16 probabilities as operands (see above)

template <typename T>
struct PrefillParams {
  const T* q;
  const T* k;
  const T* v;
  const void* mask;
  T* out;
  int64_t qs[3], ks[3], vs[3];  // batch, head, token strides (elements)
  int64_t ms[4];                // mask strides: batch, head, query, key
  int batch, q_heads, kv_heads, groups, tokens;
  int mask_dtype, causal, compat;
  float scale;
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float load_mask(const void* mask, int dtype, int64_t index) {
  if (dtype == B200_F32) return static_cast<const float*>(mask)[index];
  if (dtype == B200_F16) return __half2float(static_cast<const __half*>(mask)[index]);
  return __bfloat162float(static_cast<const __nv_bfloat16*>(mask)[index]);
}

template <bool B>
struct Flag { static constexpr bool value = B; };

template <int D>
__device__ __forceinline__ uint32_t tile_offset(int row, int chunk) {
  return static_cast<uint32_t>(row * (D * 2) + (((chunk & ~7) | ((chunk ^ row) & 7)) << 4));
}

// One output row by a whole warp, key by key, touching only the keys that the row sees: what an fp16 row is put right
// with when its tile product met an infinite or NaN value row of a key that it does not see (0 * inf; fp16
// activations do overflow). (A row that is NaN by itself, for its scores or for seeing nothing, is left alone.)
template <typename T, int D>
__device__ __noinline__ void attend_row(const PrefillParams<T>& p, int b, int hq, int qrow) {
  const int lane = threadIdx.x & 31, kvh = hq / p.groups;
  const T* q = p.q + b * p.qs[0] + hq * p.qs[1] + static_cast<int64_t>(qrow) * p.qs[2];
  float m = -INFINITY, l = 0.0f, acc[D / 32] = {};
  const int key_end = p.causal ? qrow + 1 : p.tokens;
  for (int key = 0; key < key_end; ++key) {
    const T* k = p.k + b * p.ks[0] + kvh * p.ks[1] + static_cast<int64_t>(key) * p.ks[2];
    const T* v = p.v + b * p.vs[0] + kvh * p.vs[1] + static_cast<int64_t>(key) * p.vs[2];
    float s = 0.0f;
    for (int d = lane; d < D; d += 32) s = fmaf(Elem<T>::load(q + d), Elem<T>::load(k + d), s);
    s = warp_sum(s);
    s = p.compat ? Elem<T>::round(Elem<T>::round(s) * p.scale) : s * p.scale;
    if (p.mask != nullptr)
      s += load_mask(p.mask, p.mask_dtype,
                     b * p.ms[0] + static_cast<int64_t>(qrow) * p.ms[2] + static_cast<int64_t>(key) * p.ms[3]);
    const float m_new = fmaxf(m, s), m_safe = m_new == -INFINITY ? 0.0f : m_new;
    const float alpha = expf(m - m_safe), pr = expf(s - m_safe);
    l = l * alpha + pr;
    for (int i = 0; i < D / 32; ++i) acc[i] = acc[i] * alpha + pr * Elem<T>::load(v + lane + 32 * i);
    m = m_new;
  }
  T* out = p.out + ((static_cast<int64_t>(b) * p.tokens + qrow) * p.q_heads + hq) * D;
  for (int i = 0; i < D / 32; ++i) Elem<T>::store(out + lane + 32 * i, acc[i] / l);
}

template <typename T, int D, int STAGES>
__global__ void __launch_bounds__(kThreads) prefill_attention_kernel(const PrefillParams<T> p) {
  grid_launch_dependents();
  grid_dependency_wait();
  constexpr bool kHalf = IsHalf<T>::value;
  constexpr int kChunksPerRow = D / 8;
  constexpr int kTileBytes = kBN * D * 2;
  constexpr int kQBytes = kBM * D * 2;
  constexpr int kStageBytes = 2 * kTileBytes;
  constexpr int kCopies = kBN * kChunksPerRow / kThreads;
  constexpr int kKSteps = D / 16;
  constexpr int kNTiles = D / 8;

  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t q_sm = smem_u32(smem);
  const uint32_t kv_sm = q_sm + kQBytes;

  const int q0 = blockIdx.x * kBM;
  const int hq = blockIdx.y;
  const int b = blockIdx.z;
  const int kvh = hq / p.groups;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tokens = p.tokens;

  const T* qg = p.q + b * p.qs[0] + hq * p.qs[1];
  const T* kg = p.k + b * p.ks[0] + kvh * p.ks[1];
  const T* vg = p.v + b * p.vs[0] + kvh * p.vs[1];

  const int key_end = p.causal ? min(tokens, q0 + kBM) : tokens;
  const int n_tiles = (key_end + kBN - 1) / kBN;

  auto issue_kv = [&](int tile) {
    const uint32_t kdst = kv_sm + (tile % STAGES) * kStageBytes;
    const uint32_t vdst = kdst + kTileBytes;
    const int t0 = tile * kBN;
#pragma unroll
    for (int i = 0; i < kCopies; ++i) {
      const int id = i * kThreads + threadIdx.x;
      const int r = id / kChunksPerRow, c = id % kChunksPerRow;
      const int token = t0 + r;
      const bool valid = token < tokens;
      const uint32_t soff = tile_offset<D>(r, c);
      cp_async16_zfill(kdst + soff, valid ? kg + token * p.ks[2] + c * 8 : kg, valid ? 16 : 0);
      cp_async16_zfill(vdst + soff, valid ? vg + token * p.vs[2] + c * 8 : vg, valid ? 16 : 0);
    }
  };

  // Q tile rides in the first commit group
#pragma unroll
  for (int i = 0; i < kBM * kChunksPerRow / kThreads; ++i) {
    const int id = i * kThreads + threadIdx.x;
    const int r = id / kChunksPerRow, c = id % kChunksPerRow;
    const int token = q0 + r;
    const bool valid = token < tokens;
    cp_async16_zfill(q_sm + tile_offset<D>(r, c), valid ? qg + token * p.qs[2] + c * 8 : qg,
                     valid ? 16 : 0);
  }
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < n_tiles) issue_kv(s);
    cp_async_commit();
  }

  uint32_t qa[kKSteps][4];
  float m_run[2] = {-INFINITY, -INFINITY};
  float l_run[2] = {0.0f, 0.0f};
  float oacc[kNTiles][4];
#pragma unroll
  for (int i = 0; i < kNTiles; ++i) oacc[i][0] = oacc[i][1] = oacc[i][2] = oacc[i][3] = 0.0f;

  // scores in the log2 domain (bf16) or the natural one (fp16: see the top of this file)
  constexpr float kUnit = kHalf ? 1.0f : kLog2e;
  const float scale = p.scale * kUnit;
  auto probability = [](float x) { return kHalf ? expf(x) : fast_exp2(x); };
  const int mat = lane >> 3;
  const int row_lo = q0 + warp * 16 + (lane >> 2);  // this thread's query rows: row_lo, row_lo + 8

  for (int tile = 0; tile < n_tiles; ++tile) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (tile + STAGES - 1 < n_tiles) issue_kv(tile + STAGES - 1);
    cp_async_commit();

    if (tile == 0) {
#pragma unroll
      for (int ks = 0; ks < kKSteps; ++ks) {
        const int r = warp * 16 + ((mat & 1) << 3) + (lane & 7);
        ldmatrix_x4(qa[ks], q_sm + tile_offset<D>(r, ks * 2 + (mat >> 1)));
      }
    }
    const int k0 = tile * kBN;
    // a warp whose 16 rows all precede this key tile has nothing to do under causality
    const bool warp_active = !p.causal || k0 <= q0 + warp * 16 + 15;
    if (!warp_active) continue;

    const uint32_t ksm = kv_sm + (tile % STAGES) * kStageBytes;
    const uint32_t vsm = ksm + kTileBytes;

    float sacc[kBN / 8][4];
#pragma unroll
    for (int i = 0; i < kBN / 8; ++i) sacc[i][0] = sacc[i][1] = sacc[i][2] = sacc[i][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < kKSteps; ++ks) {
#pragma unroll
      for (int np = 0; np < kBN / 16; ++np) {
        uint32_t kb[4];
        const int r = np * 16 + ((mat >> 1) << 3) + (lane & 7);
        ldmatrix_x4(kb, ksm + tile_offset<D>(r, ks * 2 + (mat & 1)));
        mma_16816<T>(sacc[np * 2], qa[ks], kb[0], kb[1]);
        mma_16816<T>(sacc[np * 2 + 1], qa[ks], kb[2], kb[3]);
      }
    }

    float row_max[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nt = 0; nt < kBN / 8; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int qrow = row_lo + ((e >> 1) << 3);
        const int key = k0 + nt * 8 + (lane & 3) * 2 + (e & 1);
        float s;
        if (p.compat)
          s = Elem<T>::round(Elem<T>::round(sacc[nt][e]) * p.scale) * kUnit;
        else
          s = sacc[nt][e] * scale;
        const bool visible = key < tokens && qrow < tokens && (!p.causal || key <= qrow);
        if (visible) {
          if (p.mask != nullptr)
            s += load_mask(p.mask, p.mask_dtype,
                           b * p.ms[0] + static_cast<int64_t>(qrow) * p.ms[2] +
                               static_cast<int64_t>(key) * p.ms[3]) *
                 kUnit;
        } else {
          s = -INFINITY;
        }
        sacc[nt][e] = s;
        row_max[e >> 1] = fmaxf(row_max[e >> 1], s);
      }
    }
    float alpha[2], m_safe[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float mx = row_max[r];
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_new = fmaxf(m_run[r], mx);
      m_safe[r] = m_new == -INFINITY ? 0.0f : m_new;
      alpha[r] = probability(m_run[r] - m_safe[r]);
      m_run[r] = m_new;
      l_run[r] *= alpha[r];
    }
    if constexpr (kHalf) {
      // the parts of 2^15 P, and the tile's part of the denominators
      uint32_t pa[kBN / 16][3][4];
      float l_tile[2] = {0.0f, 0.0f};
#pragma unroll
      for (int kk = 0; kk < kBN / 16; ++kk) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float pr[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            pr[e] = probability(sacc[kk * 2 + half][e] - m_safe[e >> 1]);
            l_tile[e >> 1] += pr[e];
            pr[e] *= kHalfScale;
          }
#pragma unroll
          for (int part = 0; part < 3; ++part) {
            const uint32_t lo = Elem<T>::pack(pr[0], pr[1]), hi = Elem<T>::pack(pr[2], pr[3]);
            pa[kk][part][half * 2] = lo;
            pa[kk][part][half * 2 + 1] = hi;
            pr[0] = (pr[0] - Elem<T>::lo(lo)) * kPartScale;
            pr[1] = (pr[1] - Elem<T>::hi(lo)) * kPartScale;
            pr[2] = (pr[2] - Elem<T>::lo(hi)) * kPartScale;
            pr[3] = (pr[3] - Elem<T>::hi(hi)) * kPartScale;
          }
        }
      }
      l_run[0] += l_tile[0];
      l_run[1] += l_tile[1];
#pragma unroll
      for (int np = 0; np < kNTiles / 2; ++np) {
        float sum[3][2][4] = {};
#pragma unroll
        for (int kk = 0; kk < kBN / 16; ++kk) {
          uint32_t vb[4];
          const int r = kk * 16 + ((mat & 1) << 3) + (lane & 7);
          ldmatrix_x4_trans(vb, vsm + tile_offset<D>(r, np * 2 + (mat >> 1)));
#pragma unroll
          for (int part = 0; part < 3; ++part) {
            mma_16816<T>(sum[part][0], pa[kk][part], vb[0], vb[1]);
            mma_16816<T>(sum[part][1], pa[kk][part], vb[2], vb[3]);
          }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float tile_sum = fmaf(fmaf(sum[2][c][e], 1.0f / kPartScale, sum[1][c][e]), 1.0f / kPartScale, sum[0][c][e]);
            oacc[np * 2 + c][e] = fmaf(oacc[np * 2 + c][e], alpha[e >> 1], tile_sum);
          }
      }
    } else {
#pragma unroll
      for (int i = 0; i < kNTiles; ++i) {
        oacc[i][0] *= alpha[0];
        oacc[i][1] *= alpha[0];
        oacc[i][2] *= alpha[1];
        oacc[i][3] *= alpha[1];
      }
#pragma unroll
      for (int kk = 0; kk < kBN / 16; ++kk) {
        uint32_t pa[4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int nt = kk * 2 + half;
          const float p0 = probability(sacc[nt][0] - m_safe[0]);
          const float p1 = probability(sacc[nt][1] - m_safe[0]);
          const float p2 = probability(sacc[nt][2] - m_safe[1]);
          const float p3 = probability(sacc[nt][3] - m_safe[1]);
          l_run[0] += p0 + p1;
          l_run[1] += p2 + p3;
          pa[half * 2] = Elem<T>::pack(p0, p1);
          pa[half * 2 + 1] = Elem<T>::pack(p2, p3);
        }
#pragma unroll
        for (int np = 0; np < kNTiles / 2; ++np) {
          uint32_t vb[4];
          const int r = kk * 16 + ((mat & 1) << 3) + (lane & 7);
          ldmatrix_x4_trans(vb, vsm + tile_offset<D>(r, np * 2 + (mat >> 1)));
          mma_16816<T>(oacc[np * 2], pa, vb[0], vb[1]);
          mma_16816<T>(oacc[np * 2 + 1], pa, vb[2], vb[3]);
        }
      }
    }
  }
  cp_async_wait<0>();

#pragma unroll
  for (int r = 0; r < 2; ++r) {
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
  }
  bool again[2] = {false, false};  // fp16: NaN, though the row sees a key and its scores are numbers
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int qrow = row_lo + r * 8;
    if (qrow >= tokens) continue;
    // all-masked row: 0 * inf = NaN, as the oracle
    const float inv = 1.0f / l_run[r];
    auto quotient = [&](float sum) { return kHalf ? sum * (1.0f / kHalfScale) / l_run[r] : sum * inv; };
    T* orow = p.out + ((static_cast<int64_t>(b) * tokens + qrow) * p.q_heads + hq) * D;
#pragma unroll
    for (int nt = 0; nt < kNTiles; ++nt) {
      const int col = nt * 8 + (lane & 3) * 2;
      const float y0 = quotient(oacc[nt][r * 2]), y1 = quotient(oacc[nt][r * 2 + 1]);
      *reinterpret_cast<uint32_t*>(orow + col) = Elem<T>::pack(y0, y1);
      again[r] = again[r] || (l_run[r] > 0.0f && (isnan(y0) || isnan(y1)));
    }
  }
  if constexpr (kHalf) {
    __syncwarp();  // the rows stored above come before those that are stored again
    for (int i = 0; i < 16; ++i)
      if (__any_sync(0xffffffffu, (lane >> 2) == (i & 7) && again[i >> 3]))
        attend_row<T, D>(p, b, hq, q0 + warp * 16 + i);
  }
}

// ---- CUDA cores: fp32, head sizes 16 / 32 / 256, fp16 without 16-byte rows ----
// fp32 arithmetic, one rounding on the way out (and, in the compatible mode of a 16-bit type, the reference's two
// roundings of the scores). A CTA of 16 x 16 threads owns 64 query rows of one (sequence, query head) and walks 64-key
// tiles: scores 4 x 4 a thread from transposed Q and K tiles, then 4 rows x D / 16 columns of P V, whose 64-key sums
// are added to the running output one tile at a time (short chains: rounding errors grow with the tiles, not the keys).
// A key that a row does not see has probability -1 and is skipped: its value may be infinite or NaN. Bound by the FMA
// rate (4 FMA a shared-memory word) and by the few CTAs of a short prompt.
// Qwen2-0.5B in fp32, 1 x 1000 tokens: 126.8 -> 34.4 ms a pass with the tiled GEMM of linear.cu (before: one CTA per
// query row, every row reading all keys and values again).
template <int D>
constexpr int kTiledSmem = (2 * D * 68 + 64 * D + 64 * 68) * 4;

template <int D, typename T, bool VEC>
__global__ void __launch_bounds__(256) prefill_attention_tiled_kernel(const PrefillParams<T> p) {
  constexpr int kPitch = 68, kColumns = D / 16;
  extern __shared__ __align__(16) float tiled_smem[];
  float* q_sm = tiled_smem;              // [D][68]: Q transposed
  float* k_sm = q_sm + D * kPitch;       // [D][68]: K transposed
  float* v_sm = k_sm + D * kPitch;       // [64][D]
  float* p_sm = v_sm + 64 * D;           // [64 keys][68 rows]
  const int q0 = blockIdx.x * 64, hq = blockIdx.y, b = blockIdx.z, kvh = hq / p.groups;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const T* q = p.q + b * p.qs[0] + hq * p.qs[1];
  const T* k = p.k + b * p.ks[0] + kvh * p.ks[1];
  const T* v = p.v + b * p.vs[0] + kvh * p.vs[1];

  // 64 rows from `first` on, zeros behind the last token
  auto load_rows = [&](const T* base, int64_t stride, int first, float* to, bool transposed) {
    constexpr int kVec = VEC ? Elem<T>::kPerVec : 1;
    for (int at = threadIdx.x * kVec; at < 64 * D; at += 256 * kVec) {
      const int row = at / D, d = at % D;
      float value[kVec];
      if (first + row >= p.tokens) {
#pragma unroll
        for (int e = 0; e < kVec; ++e) value[e] = 0.0f;
      } else if constexpr (VEC) {
        Vec16<T> raw;
        raw.load(base + (first + row) * stride + d);
#pragma unroll
        for (int e = 0; e < kVec; ++e) value[e] = raw.v[e];
      } else {
        value[0] = Elem<T>::load(base + (first + row) * stride + d);
      }
#pragma unroll
      for (int e = 0; e < kVec; ++e) to[transposed ? (d + e) * kPitch + row : row * D + d + e] = value[e];
    }
  };

  load_rows(q, p.qs[2], q0, q_sm, true);
  float m[4], l[4], out[4][kColumns];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.0f;
#pragma unroll
    for (int c = 0; c < kColumns; ++c) out[i][c] = 0.0f;
  }
  const int key_end = p.causal ? min(p.tokens, q0 + 64) : p.tokens;
  for (int k0 = 0; k0 < key_end; k0 += 64) {
    __syncthreads();  // the last tile's products have read K, V and P
    load_rows(k, p.ks[2], k0, k_sm, true);
    load_rows(v, p.vs[2], k0, v_sm, false);
    __syncthreads();
    float s[4][4] = {};
#pragma unroll 4
    for (int d = 0; d < D; ++d) {
      const float4 a = *reinterpret_cast<const float4*>(q_sm + d * kPitch + ty * 4);
      const float4 c = *reinterpret_cast<const float4*>(k_sm + d * kPitch + tx * 4);
      const float av[4] = {a.x, a.y, a.z, a.w}, cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = fmaf(av[i], cv[j], s[i][j]);
    }
    const bool whole = k0 + 64 <= p.tokens && (!p.causal || k0 + 63 <= q0);  // every row sees every key
    float alpha[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = q0 + ty * 4 + i;
      bool seen[4];
      float top = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = k0 + tx * 4 + j;
        seen[j] = whole || (key < p.tokens && (!p.causal || key <= row));
        s[i][j] = p.compat ? Elem<T>::round(Elem<T>::round(s[i][j]) * p.scale) : s[i][j] * p.scale;
        if (p.mask != nullptr && seen[j] && row < p.tokens)
          s[i][j] += load_mask(p.mask, p.mask_dtype,
                               b * p.ms[0] + static_cast<int64_t>(row) * p.ms[2] + static_cast<int64_t>(key) * p.ms[3]);
        if (seen[j]) top = fmaxf(top, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      const float m_new = fmaxf(m[i], top), m_safe = m_new == -INFINITY ? 0.0f : m_new;
      alpha[i] = expf(m[i] - m_safe);
      m[i] = m_new;
      float sum = 0.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = seen[j] ? expf(s[i][j] - m_safe) : -1.0f;
        sum += seen[j] ? s[i][j] : 0.0f;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l[i] = l[i] * alpha[i] + sum;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<float4*>(p_sm + (tx * 4 + j) * kPitch + ty * 4) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
    __syncthreads();
    float part[4][kColumns] = {};
    const int keys = min(64, key_end - k0);
    auto add_keys = [&](auto masked) {
      const int end = decltype(masked)::value ? keys : 64;  // (a tile that every row sees whole has them all)
#pragma unroll 4
      for (int key = 0; key < end; ++key) {
        const float4 w = *reinterpret_cast<const float4*>(p_sm + key * kPitch + ty * 4);
        const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int c = 0; c < kColumns; ++c) {
          const float value = v_sm[key * D + tx + 16 * c];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float next = fmaf(wv[i], value, part[i][c]);
            part[i][c] = decltype(masked)::value && wv[i] < 0.0f ? part[i][c] : next;
          }
        }
      }
    };
    if (whole) add_keys(Flag<false>{});
    else add_keys(Flag<true>{});
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < kColumns; ++c) out[i][c] = out[i][c] * alpha[i] + part[i][c];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = q0 + ty * 4 + i;
    if (row >= p.tokens) continue;
    T* to = p.out + ((static_cast<int64_t>(b) * p.tokens + row) * p.q_heads + hq) * D;
#pragma unroll
    for (int c = 0; c < kColumns; ++c) Elem<T>::store(to + tx + 16 * c, out[i][c] / l[i]);
  }
}

// The same for a few query rows of a few keys, which leave a tile mostly empty: one CTA per row, thread t owning the keys
// t, t + 64, ... with an online softmax of its own; the CTA merges. Bound by latency: 14 heads of 64 in fp32, 4, 16, 32
// tokens 5.0, 6.9, 10.0 us against 9.2, 9.8, 10.9 in tiles; 64 tokens 25.7 against 13.4.
template <int D, typename T>
__global__ void __launch_bounds__(64) prefill_attention_rows_kernel(const PrefillParams<T> p) {
  constexpr int kThreadsOfRow = 64;
  const int qrow = blockIdx.x, hq = blockIdx.y, b = blockIdx.z, kvh = hq / p.groups;
  __shared__ float sq[D], sm[kThreadsOfRow], sl[kThreadsOfRow];
  __shared__ float so[kThreadsOfRow][D + 1];
  for (int d = threadIdx.x; d < D; d += kThreadsOfRow)
    sq[d] = Elem<T>::load(p.q + b * p.qs[0] + hq * p.qs[1] + qrow * p.qs[2] + d);
  __syncthreads();
  float m = -INFINITY, l = 0.0f, acc[D];
#pragma unroll
  for (int d = 0; d < D; ++d) acc[d] = 0.0f;
  const int key_end = p.causal ? qrow + 1 : p.tokens;
  for (int t = threadIdx.x; t < key_end; t += kThreadsOfRow) {
    const T* key = p.k + b * p.ks[0] + kvh * p.ks[1] + t * p.ks[2];
    const T* value = p.v + b * p.vs[0] + kvh * p.vs[1] + t * p.vs[2];
    float s = 0.0f;
#pragma unroll
    for (int d = 0; d < D; ++d) s = fmaf(sq[d], Elem<T>::load(key + d), s);
    s = p.compat ? Elem<T>::round(Elem<T>::round(s) * p.scale) : s * p.scale;
    if (p.mask != nullptr)
      s += load_mask(p.mask, p.mask_dtype, b * p.ms[0] + static_cast<int64_t>(qrow) * p.ms[2] + t * p.ms[3]);
    const float m_new = fmaxf(m, s), m_safe = m_new == -INFINITY ? 0.0f : m_new;
    const float alpha = expf(m - m_safe), pr = expf(s - m_safe);
    l = l * alpha + pr;
#pragma unroll
    for (int d = 0; d < D; ++d) acc[d] = acc[d] * alpha + pr * Elem<T>::load(value + d);
    m = m_new;
  }
  sm[threadIdx.x] = m;
  sl[threadIdx.x] = l;
#pragma unroll
  for (int d = 0; d < D; ++d) so[threadIdx.x][d] = acc[d];
  __syncthreads();
  const int used = min(kThreadsOfRow, key_end);  // threads that had a key
  for (int d = threadIdx.x; d < D; d += kThreadsOfRow) {
    float m_all = -INFINITY, l_all = 0.0f, o_all = 0.0f;
    for (int t = 0; t < used; ++t) m_all = fmaxf(m_all, sm[t]);
    for (int t = 0; t < used; ++t) {
      // (a thread whose keys are all hidden weighs nothing; its sums may be NaN, as 0 * inf is, and count)
      const float weight = sm[t] == -INFINITY ? 0.0f : expf(sm[t] - m_all);
      l_all += sl[t] * weight;
      o_all += so[t][d] * weight;
    }
    Elem<T>::store(p.out + ((static_cast<int64_t>(b) * p.tokens + qrow) * p.q_heads + hq) * D + d, o_all / l_all);
  }
}

template <int D, typename T>
int launch_row_by_row(const PrefillParams<T>& p, cudaStream_t stream) {
  prefill_attention_rows_kernel<D, T><<<dim3(p.tokens, p.q_heads, p.batch), 64, 0, stream>>>(p);
  return launch_status();
}

template <int D, typename T>
int launch_tiled(const PrefillParams<T>& p, bool vec, cudaStream_t stream) {
  auto launch = [&](auto kernel) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTiledSmem<D>) != cudaSuccess)
      return B200_ERR_LAUNCH;
    kernel<<<dim3((p.tokens + 63) / 64, p.q_heads, p.batch), 256, kTiledSmem<D>, stream>>>(p);
    return launch_status();
  };
  return vec ? launch(prefill_attention_tiled_kernel<D, T, true>) : launch(prefill_attention_tiled_kernel<D, T, false>);
}

template <int D, int STAGES, typename T>
int launch_warp_level(const PrefillParams<T>& p, cudaStream_t stream) {
  constexpr int smem = kBM * D * 2 + STAGES * 2 * kBN * D * 2;
  auto kernel = prefill_attention_kernel<T, D, STAGES>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return B200_ERR_LAUNCH;
  dim3 grid((p.tokens + kBM - 1) / kBM, p.q_heads, p.batch);
  return launch_chained(kernel, grid, dim3(kThreads), smem, stream, p) == cudaSuccess ? launch_status() : B200_ERR_LAUNCH;
}

}  // namespace
}  // namespace b200

namespace b200 {
// prefill_attention_tcgen05.cu
int prefill_attention_tcgen05(const void* query, const void* key, const void* value, void* output,
                              int64_t batch, int64_t q_heads, int64_t kv_heads, int64_t tokens,
                              int64_t head_dim, const int64_t query_strides[4],
                              const int64_t key_strides[4], const int64_t value_strides[4],
                              double scale, int32_t* status, cudaStream_t stream, const void* mask,
                              const int64_t* mask_strides, void* workspace, int64_t workspace_bytes,
                              int64_t context, const void* sink, int64_t chunk);
int64_t prefill_attention_tcgen05_workspace_bytes(int64_t batch, int64_t tokens);
}  // namespace b200

using namespace b200;

extern "C" int64_t b200_prefill_attention_workspace_bytes(int64_t batch, int64_t tokens) {
  if (batch <= 0 || tokens <= 0) return 0;
  return prefill_attention_tcgen05_workspace_bytes(batch, tokens);
}

extern "C" int b200_prefill_attention(const void* query, const void* key, const void* value,
                                      const void* mask, void* output, int64_t batch,
                                      int64_t q_heads, int64_t kv_heads, int64_t tokens,
                                      int64_t head_dim, const int64_t query_strides[4],
                                      const int64_t key_strides[4],
                                      const int64_t value_strides[4],
                                      const int64_t mask_strides[4], int mask_dtype, double scale,
                                      int causal, int dtype, int mode, void* workspace,
                                      int64_t workspace_bytes, int32_t* status, void* stream) {
  if (!query || !key || !value || !output || !query_strides || !key_strides || !value_strides ||
      batch < 0 || q_heads <= 0 || kv_heads <= 0 || tokens < 0 || head_dim <= 0 ||
      q_heads % kv_heads != 0)
    return B200_ERR_BAD_ARGUMENT;
  if (mask == nullptr && !causal) return B200_ERR_BAD_ARGUMENT;
  if (mask != nullptr && (!mask_strides || (!known_dtype(mask_dtype))))
    return B200_ERR_BAD_ARGUMENT;
  if (query_strides[3] != 1 || key_strides[3] != 1 || value_strides[3] != 1)
    return B200_ERR_UNSUPPORTED;
  if (batch == 0 || tokens == 0) return B200_OK;
  if (batch > 65535 || q_heads > 65535 || tokens > INT32_MAX) return B200_ERR_TOO_LARGE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int groups = static_cast<int>(q_heads / kv_heads);
  const int64_t zero4[4] = {0, 0, 0, 0};
  const int64_t* ms = mask != nullptr ? mask_strides : zero4;

  if (!known_dtype(dtype)) return B200_ERR_UNSUPPORTED;
  // 16-byte loads of every row: what the tensor-core kernels need (bf16 is refused without them, fp16 then takes the
  // CUDA-core kernel)
  const int per_vec = dtype == B200_F32 ? 4 : 8;
  bool rows16 = aligned16(query) && aligned16(key) && aligned16(value);
  for (int i = 0; i < 3; ++i)
    rows16 = rows16 && query_strides[i] % per_vec == 0 && key_strides[i] % per_vec == 0 && value_strides[i] % per_vec == 0;
  const bool pairs = (reinterpret_cast<uintptr_t>(output) & 3u) == 0;
  // A few rows of a few keys are faster row by row, not in tiles. The line lies where the tiles win, us row by row and in
  // tiles: fp32, heads of 64, 4 heads x 48 tokens 10.9 and 12.1, x 96 21.5 and 20.0; 28 heads x 16 tokens 7.4 and 10.0, x
  // 24 10.8 and 10.3; heads of 128, 14 heads x 16 tokens 11.9 and 16.4, x 32 18.3 and 17.5; fp16, heads of 32, 4 heads x
  // 128 tokens 12.4 and 12.8; heads of 16, 4 heads x 128 tokens 8.7 and 10.3. fp16 on the tensor cores: 14 heads of 64, 8
  // tokens 5.0 and 6.3, 32 tokens 6 and 7.
  const bool few = head_dim <= 128 && tokens * head_dim <= 4096 && batch * q_heads * tokens <= 512;
  const bool tensor_core = (head_dim == 64 || head_dim == 128) &&
                           (dtype == B200_BF16 || (dtype == B200_F16 && rows16 && pairs && !(few && tokens <= 8)));
  if (!tensor_core) {
    if (head_dim != 16 && head_dim != 32 && head_dim != 64 && head_dim != 128 && head_dim != 256)
      return B200_ERR_UNSUPPORTED;
    if (tokens > 65535 * 64) return B200_ERR_TOO_LARGE;
  } else {
    if (!rows16 || !pairs) return B200_ERR_ALIGNMENT;
    if (dtype == B200_BF16 && mode == B200_MODE_FAST &&
        ((mask == nullptr && causal) ||
         (mask != nullptr && !causal && mask_dtype == B200_F32 && workspace != nullptr))) {
      // the tensor-core kernel: causal-proved, or the additive-mask contract with its tile pre-pass
      const int code = prefill_attention_tcgen05(query, key, value, output, batch, q_heads, kv_heads,
                                                 tokens, head_dim, query_strides, key_strides,
                                                 value_strides, scale, status, s, mask, mask_strides,
                                                 workspace, workspace_bytes, 0, nullptr, 0);
      if (code != B200_ERR_UNSUPPORTED) return code;
    }
  }

  int code = B200_ERR_UNSUPPORTED;
  with_element_type(dtype, [&](auto tag) {
    using T = typename decltype(tag)::type;
    PrefillParams<T> p;
    p.q = static_cast<const T*>(query);
    p.k = static_cast<const T*>(key);
    p.v = static_cast<const T*>(value);
    p.mask = mask;
    p.out = static_cast<T*>(output);
    for (int i = 0; i < 3; ++i) {
      p.qs[i] = query_strides[i];
      p.ks[i] = key_strides[i];
      p.vs[i] = value_strides[i];
    }
    for (int i = 0; i < 4; ++i) p.ms[i] = ms[i];
    p.batch = static_cast<int>(batch);
    p.q_heads = static_cast<int>(q_heads);
    p.kv_heads = static_cast<int>(kv_heads);
    p.groups = groups;
    p.tokens = static_cast<int>(tokens);
    p.mask_dtype = mask_dtype;
    p.causal = causal ? 1 : 0;
    p.compat = mode == B200_MODE_PYTORCH_COMPATIBLE && dtype != B200_F32 ? 1 : 0;
    p.scale = static_cast<float>(scale);
    if constexpr (sizeof(T) == 2) {
      if (tensor_core) {
        code = head_dim == 64 ? launch_warp_level<64, 3>(p, s) : launch_warp_level<128, 2>(p, s);
        return;
      }
    }
    if (few) {
      if (head_dim == 16) code = launch_row_by_row<16>(p, s);
      else if (head_dim == 32) code = launch_row_by_row<32>(p, s);
      else if (head_dim == 64) code = launch_row_by_row<64>(p, s);
      else code = launch_row_by_row<128>(p, s);
      return;
    }
    if (head_dim == 16) code = launch_tiled<16>(p, rows16, s);
    else if (head_dim == 32) code = launch_tiled<32>(p, rows16, s);
    else if (head_dim == 64) code = launch_tiled<64>(p, rows16, s);
    else if (head_dim == 128) code = launch_tiled<128>(p, rows16, s);
    else code = launch_tiled<256>(p, rows16, s);
  });
  return code;
}
