// serve.linear: y[M,N] = x[M,K] W[N,K]^T (+ bias) with fp32 accumulation and fused
// epilogues (residual add, SwiGLU over row-interleaved gate/up weights).
//
// bf16, fp16: warp-level tensor-core tiles (m16n8k16) fed by a multi-stage cp.async ring of
// 128-byte XOR-swizzled rows. Both operands are K-major, so A (activations) and B
// (weights) are read with plain ldmatrix. Decode-sized M streams every weight byte
// exactly once; when the tile grid is smaller than ~2 waves of the 148 SMs the K range
// is split across CTAs (grid.z): each CTA parks its fp32 partial in the workspace and the
// CTA that arrives last at the tile's counter adds the partials in split order
// (deterministic) and runs the epilogue. Counters are left at zero for the next call.
//
// fp32, and fp16 whose K or rows do not allow 16-byte copies: CUDA-core tiled GEMM with IEEE fp32 FMAs.
#include <stdlib.h>
#include <string.h>

#include "common.cuh"

namespace b200 {
namespace {

constexpr int kBK = 64;  // 16-bit K extent of a stage: 128-byte rows

template <typename T>
struct LinearParams {
  const T* x;
  const T* w;
  const T* bias;
  const T* residual;
  T* out;
  float* partials;
  int* counters;
  int64_t x_row_stride;
  int m, k, n, splits, epilogue;
};

__device__ __forceinline__ float silu_f32(float x) {
  return __fdiv_rn(x, __fadd_rn(1.0f, expf(-x)));
}

// Writes the pair of adjacent columns (n, n+1) of row m.
template <typename T>
__device__ __forceinline__ void epilogue_pair(const LinearParams<T>& p, int m, int n, float v0,
                                              float v1) {
  if (m >= p.m || n >= p.n) return;
  const bool has1 = n + 1 < p.n;
  if (p.bias != nullptr) {
    v0 += Elem<T>::load(p.bias + n);
    if (has1) v1 += Elem<T>::load(p.bias + n + 1);
  }
  if (p.epilogue == B200_EPILOGUE_SWIGLU) {
    // column 2j is gate_j, column 2j+1 is up_j
    const float g = Elem<T>::round(silu_f32(Elem<T>::round(v0)));
    const float u = Elem<T>::round(v1);
    Elem<T>::store(p.out + static_cast<int64_t>(m) * (p.n / 2) + n / 2, g * u);
    return;
  }
  v0 = Elem<T>::round(v0);
  v1 = Elem<T>::round(v1);
  const int64_t o = static_cast<int64_t>(m) * p.n + n;
  if (p.epilogue == B200_EPILOGUE_RESIDUAL) {
    v0 = __fadd_rn(v0, Elem<T>::load(p.residual + o));
    if (has1) v1 = __fadd_rn(v1, Elem<T>::load(p.residual + o + 1));
  }
  if (has1 && (reinterpret_cast<uintptr_t>(p.out + o) & 3u) == 0) {
    *reinterpret_cast<uint32_t*>(p.out + o) = Elem<T>::pack(v0, v1);
  } else {
    Elem<T>::store(p.out + o, v0);
    if (has1) Elem<T>::store(p.out + o + 1, v1);
  }
}

template <typename T, int BM, int BN, int WM, int WN, int STAGES>
__global__ void __launch_bounds__(WM* WN * 32) linear_warp_kernel(const LinearParams<T> p) {
  constexpr int kThreads = WM * WN * 32;
  constexpr int WTM = BM / WM, WTN = BN / WN;
  constexpr int MT = WTM / 16, NT = WTN / 8;
  static_assert(WTM % 16 == 0 && WTN % 16 == 0, "warp tile must be a multiple of 16 x 16");
  constexpr int kABytes = BM * 128, kBBytes = BN * 128, kStageBytes = kABytes + kBBytes;
  constexpr int kAcc = MT * NT * 4;

  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t smem_base = smem_u32(smem);

  const int tile_n = blockIdx.x, tile_m = blockIdx.y, split = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warp_m = warp / WN, warp_n = warp % WN;

  const int kb_total = (p.k + kBK - 1) / kBK;
  const int kb_per = (kb_total + p.splits - 1) / p.splits;
  const int kb0 = split * kb_per;
  const int nkb = max(0, min(kb0 + kb_per, kb_total) - kb0);

  auto issue_load = [&](int stage, int kb) {
    const uint32_t a_dst = smem_base + stage * kStageBytes;
    const uint32_t b_dst = a_dst + kABytes;
    const int k0 = kb * kBK;
#pragma unroll
    for (int i = 0; i < (BM * 8 + kThreads - 1) / kThreads; ++i) {
      const int id = i * kThreads + threadIdx.x;
      if (BM * 8 % kThreads != 0 && id >= BM * 8) break;
      const int r = id >> 3, c = id & 7;
      const int m = tile_m * BM + r;
      const bool valid = m < p.m && k0 + c * 8 < p.k;
      const T* src = valid ? p.x + static_cast<int64_t>(m) * p.x_row_stride + k0 + c * 8 : p.x;
      cp_async16_zfill(a_dst + r * 128 + (swizzle128(r, c) << 4), src, valid ? 16 : 0);
    }
#pragma unroll
    for (int i = 0; i < (BN * 8 + kThreads - 1) / kThreads; ++i) {
      const int id = i * kThreads + threadIdx.x;
      if (BN * 8 % kThreads != 0 && id >= BN * 8) break;
      const int r = id >> 3, c = id & 7;
      const int n = tile_n * BN + r;
      const bool valid = n < p.n && k0 + c * 8 < p.k;
      const T* src = valid ? p.w + static_cast<int64_t>(n) * p.k + k0 + c * 8 : p.w;
      cp_async16_zfill(b_dst + r * 128 + (swizzle128(r, c) << 4), src, valid ? 16 : 0);
    }
  };

  float acc[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0f;

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nkb) issue_load(s, kb0 + s);
    cp_async_commit();
  }

  const int mat = lane >> 3;
  for (int i = 0; i < nkb; ++i) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (i + STAGES - 1 < nkb) issue_load((i + STAGES - 1) % STAGES, kb0 + i + STAGES - 1);
    cp_async_commit();

    const uint32_t a_sm = smem_base + (i % STAGES) * kStageBytes;
    const uint32_t b_sm = a_sm + kABytes;
#pragma unroll
    for (int ks = 0; ks < kBK / 16; ++ks) {
      uint32_t af[MT][4];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const int r = warp_m * WTM + mt * 16 + ((mat & 1) << 3) + (lane & 7);
        ldmatrix_x4(af[mt], a_sm + r * 128 + (swizzle128(r, ks * 2 + (mat >> 1)) << 4));
      }
#pragma unroll
      for (int np = 0; np < NT / 2; ++np) {
        uint32_t bf[4];
        const int r = warp_n * WTN + np * 16 + ((mat >> 1) << 3) + (lane & 7);
        ldmatrix_x4(bf, b_sm + r * 128 + (swizzle128(r, ks * 2 + (mat & 1)) << 4));
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          mma_16816<T>(acc[mt][np * 2], af[mt], bf[0], bf[1]);
          mma_16816<T>(acc[mt][np * 2 + 1], af[mt], bf[2], bf[3]);
        }
      }
    }
  }
  cp_async_wait<0>();

  if (p.splits > 1) {
    const int tile = tile_m * gridDim.x + tile_n;
    float* mine = p.partials + (static_cast<int64_t>(tile) * p.splits + split) * (kAcc * kThreads);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          mine[((mt * NT + nt) * 4 + e) * kThreads + threadIdx.x] = acc[mt][nt][e];
    __threadfence();
    __syncthreads();
    __shared__ int is_last;
    if (threadIdx.x == 0) {
      const int arrived = atomicAdd(p.counters + tile, 1);
      is_last = arrived == p.splits - 1;
      if (is_last) p.counters[tile] = 0;  // ready for the next call on this workspace
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    const float* all = p.partials + static_cast<int64_t>(tile) * p.splits * (kAcc * kThreads);
    // split-major, with all kAcc loads of a split in flight together: the sum order is fixed
    // (split 0, 1, ...), the latency of a round is paid once per split, not once per element
    float* flat = &acc[0][0][0];
    for (int s = 0; s < p.splits; ++s) {
      float part[kAcc];
#pragma unroll
      for (int i = 0; i < kAcc; ++i)
        part[i] = __ldcg(all + (static_cast<int64_t>(s) * kAcc + i) * kThreads + threadIdx.x);
#pragma unroll
      for (int i = 0; i < kAcc; ++i) flat[i] = s == 0 ? part[i] : flat[i] + part[i];
    }
  }

#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    const int m0 = tile_m * BM + warp_m * WTM + mt * 16 + (lane >> 2);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int n0 = tile_n * BN + warp_n * WTN + nt * 8 + (lane & 3) * 2;
      epilogue_pair(p, m0, n0, acc[mt][nt][0], acc[mt][nt][1]);
      epilogue_pair(p, m0 + 8, n0, acc[mt][nt][2], acc[mt][nt][3]);
    }
  }
}

// ------------------------------------------------------- CUDA cores: fp32, fp16 ----
// fp32 arithmetic for fp32 tensors and for the fp16 calls that the tensor-core kernels do not take; a 16-bit type is
// rounded where the reference's kernels round theirs (the result, the sum in front of a residual add, gate / up /
// silu(gate) of a SwiGLU). Two kernels: a few rows stream W (linear_rows_kernel), more rows are a tiled product.
template <typename T>
struct LinearParamsGeneric {
  const T* x;
  const T* w;
  const T* bias;
  const T* residual;
  T* out;
  int64_t x_row_stride;
  int m, k, n, epilogue;
  // RMS norm in front of the projection (linear_rows_kernel): x is the row before the norm
  const T* norm_weight = nullptr;
  float norm_eps = 0.0f;
};

// One output, or with SwiGLU the output of the column pair (n, n + 1): v0 is column n's sum, v1 column n + 1's.
template <typename T>
__device__ __forceinline__ void epilogue_generic(const LinearParamsGeneric<T>& p, int m, int n, float v0, float v1) {
  if (m >= p.m || n >= p.n) return;
  if (p.bias != nullptr) v0 += Elem<T>::load(p.bias + n);
  if (p.epilogue == B200_EPILOGUE_SWIGLU) {
    if (n & 1) return;
    if (p.bias != nullptr) v1 += Elem<T>::load(p.bias + n + 1);
    const float gate = Elem<T>::round(silu_f32(Elem<T>::round(v0)));
    Elem<T>::store(p.out + static_cast<int64_t>(m) * (p.n / 2) + n / 2, gate * Elem<T>::round(v1));
    return;
  }
  const int64_t o = static_cast<int64_t>(m) * p.n + n;
  if (p.epilogue == B200_EPILOGUE_RESIDUAL) v0 = __fadd_rn(Elem<T>::round(v0), Elem<T>::load(p.residual + o));
  Elem<T>::store(p.out + o, v0);
}

// fp32, up to 8 rows of x per CTA: bound by reading W once, and in a chain of launches by the time until W flows. As in
// linear_rows.cu W travels as early as it can (before the dependency wait, where the caller promises constant weights):
// every lane copies the pieces that it will multiply (cp.async) into a ring of its own, 8 columns x 4 k of a chunk of
// 128 k, so that many CTAs with few registers keep their loads in flight and the main loop has no barrier. The warps of
// a CTA (and, with few columns, of a cluster) share the K range; x comes out of L1. The sums are short chains
// (4 K / 128 / warps terms a lane) joined by a tree of exchanges in which every lane ends up with one output.
// In a chain of launches, 4 rows, against W in registers behind the launch: 9728 x 896 16.1 -> 8.4 us (4.2 TB/s), 896 x
// 4864 9.2 -> 6.3, 896 x 896 4.9 -> 2.4, LM head 151936 x 896 128 -> 83 (6.6 TB/s). 8 rows: 11.7, 7.7, 3.0, 121 (FMAs).
constexpr int kRowsWarps = 4, kRowsThreads = kRowsWarps * 32, kRowsColumns = 8, kRowsOfX = 8, kRowsRing = 4;
constexpr int kRowsChunk = 128, kRowsChunkBytes = kRowsColumns * 512;  // k, and bytes of a warp's piece of W

// Lane i's return value: the sum over the lanes of their v[i].
__device__ __forceinline__ float sum_transposed(float (&v)[32], int lane) {
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const bool upper = (lane & s) != 0;
#pragma unroll
    for (int i = 0; i < s; ++i) {
      const float given = upper ? v[i] : v[i + s], kept = upper ? v[i + s] : v[i];
      v[i] = kept + __shfl_xor_sync(0xffffffffu, given, s);
    }
  }
  return v[0];
}

//
// NORM: the RMS norm in front of the projection as well. A row's factor rsqrt(mean(x^2) + eps) does not depend on k, so
// the products take x times the norm's weight, every CTA adds the squares of the x that it reads anyway, and the factor
// scales the sums: no launch for the norm, and none of its round trips (where that pays: norm_pays_inside).
//
// ROWS: rows of x a CTA takes (4 or 8)
template <int ROWS, bool NORM>
__global__ void __launch_bounds__(kRowsThreads) linear_rows_kernel(const LinearParamsGeneric<float> p, int slots, int early) {
  extern __shared__ __align__(16) unsigned char rows_ring[];  // [warp][chunk][column][lane]
  constexpr int kOutputs = ROWS * kRowsColumns;
  __shared__ float part[kRowsWarps][kOutputs];
  __shared__ float total[kOutputs];
  __shared__ float part_squares[kRowsWarps][ROWS];
  __shared__ float total_squares[ROWS];
  grid_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * kRowsColumns, m0 = blockIdx.y * ROWS, rows = min(ROWS, p.m - m0);
  const int splits = gridDim.z, rank = blockIdx.z;
  const int chunks = (p.k + kRowsChunk - 1) / kRowsChunk, parts = splits * kRowsWarps, mine = rank * kRowsWarps + warp;
  const int first = static_cast<int>(static_cast<int64_t>(chunks) * mine / parts);
  const int count = static_cast<int>(static_cast<int64_t>(chunks) * (mine + 1) / parts) - first;
  const uint32_t base = smem_u32(rows_ring) + warp * slots * kRowsChunkBytes + lane * 16;
  // (pieces beyond K become zeros; columns beyond N repeat the last one and are not stored)
  auto copy = [&](int c) {
    if (c >= count) return;
    const int k = (first + c) * kRowsChunk + lane * 4;
    const bool there = k < p.k;  // (K is a multiple of 4)
    const uint32_t at = base + c % kRowsRing * kRowsChunkBytes;
#pragma unroll
    for (int j = 0; j < kRowsColumns; ++j)
      cp_async16_zfill(at + j * 512, p.w + static_cast<int64_t>(min(n0 + j, p.n - 1)) * p.k + (there ? k : 0), there ? 16 : 0);
  };
  if (!early) grid_dependency_wait();
#pragma unroll
  for (int c = 0; c < kRowsRing; ++c) {
    copy(c);
    cp_async_commit();
  }
  if (early) grid_dependency_wait();

  float acc[ROWS][kRowsColumns] = {};
  float squares[ROWS] = {};
  const float* x = p.x + m0 * p.x_row_stride;
  for (int c = 0; c < count; ++c) {
    const int k = (first + c) * kRowsChunk + lane * 4;
    float4 xv[ROWS], scale = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (NORM && k < p.k)
      asm volatile("ld.global.ca.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(scale.x), "=f"(scale.y), "=f"(scale.z), "=f"(scale.w)
                   : "l"(p.norm_weight + k) : "memory");
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      xv[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (i < rows && k < p.k)
        asm volatile("ld.global.ca.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(xv[i].x), "=f"(xv[i].y), "=f"(xv[i].z), "=f"(xv[i].w)
                     : "l"(x + i * p.x_row_stride + k) : "memory");
    }
    if (NORM) {
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        squares[i] = fmaf(xv[i].w, xv[i].w, fmaf(xv[i].z, xv[i].z, fmaf(xv[i].y, xv[i].y, fmaf(xv[i].x, xv[i].x, squares[i]))));
        xv[i].x *= scale.x; xv[i].y *= scale.y; xv[i].z *= scale.z; xv[i].w *= scale.w;
      }
    }
    cp_async_wait<kRowsRing - 1>();
    const uint32_t at = base + c % kRowsRing * kRowsChunkBytes;
#pragma unroll
    for (int j = 0; j < kRowsColumns; ++j) {
      float4 w;
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(w.x), "=f"(w.y), "=f"(w.z), "=f"(w.w)
                   : "r"(at + j * 512) : "memory");
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
        acc[i][j] = fmaf(xv[i].w, w.w, fmaf(xv[i].z, w.z, fmaf(xv[i].y, w.y, fmaf(xv[i].x, w.x, acc[i][j]))));
    }
    copy(c + kRowsRing);  // (every lane refills the pieces that it has read itself)
    cp_async_commit();
  }
  cp_async_wait<0>();
#pragma unroll
  for (int h = 0; h < kOutputs / 32; ++h) {
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = acc[(h * 32 + i) / kRowsColumns][i % kRowsColumns];
    part[warp][h * 32 + lane] = sum_transposed(v, lane);
  }
  if (NORM) {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const float sum = warp_sum(squares[i]);
      if (lane == 0) part_squares[warp][i] = sum;
    }
  }
  __syncthreads();
  if (splits > 1) {
    if (NORM && threadIdx.x < ROWS) {
      float sum = 0.0f;
#pragma unroll
      for (int s = 0; s < kRowsWarps; ++s) sum += part_squares[s][threadIdx.x];
      total_squares[threadIdx.x] = sum;
    }
    if (threadIdx.x < kOutputs) {
      float sum = 0.0f;
#pragma unroll
      for (int s = 0; s < kRowsWarps; ++s) sum += part[s][threadIdx.x];
      total[threadIdx.x] = sum;
    }
    cluster_sync();
  }
  // pairs of neighbouring columns, dealt to the CTAs of the cluster; sums in warp and rank order
  for (int u = rank + splits * threadIdx.x; u < kOutputs / 2; u += splits * kRowsThreads) {
    const int i = u / (kRowsColumns / 2), c = u % (kRowsColumns / 2) * 2, at = i * kRowsColumns + c;
    if (i >= rows) continue;
    float v0 = 0.0f, v1 = 0.0f;
    if (splits > 1) {
      for (int s = 0; s < splits; ++s) {
        v0 += load_cluster_f32(smem_u32(&total[at]), s);
        v1 += load_cluster_f32(smem_u32(&total[at + 1]), s);
      }
    } else {
#pragma unroll
      for (int s = 0; s < kRowsWarps; ++s) {
        v0 += part[s][at];
        v1 += part[s][at + 1];
      }
    }
    if (NORM) {
      float sum = 0.0f;
      if (splits > 1) {
        for (int s = 0; s < splits; ++s) sum += load_cluster_f32(smem_u32(&total_squares[i]), s);
      } else {
#pragma unroll
        for (int s = 0; s < kRowsWarps; ++s) sum += part_squares[s][i];
      }
      const float factor = rsqrtf(sum / static_cast<float>(p.k) + p.norm_eps);
      v0 *= factor;
      v1 *= factor;
    }
    epilogue_generic(p, m0 + i, n0 + c, v0, v1);
    epilogue_generic(p, m0 + i, n0 + c + 1, v1, 0.0f);
  }
  if (splits > 1) cluster_sync();  // no CTA leaves while another reads its sums
}

// Tiled product: 64 x 64 outputs a CTA, 4 x 8 a thread, K in blocks of 16 whose sums are added to the accumulators
// (rounding errors grow with K / 16 + 16, not with K). The next block travels in registers while this one is
// multiplied. Where the tiles are fewer than the SMs, the K range is cut over the CTAs of a cluster (up to 8 along
// grid z), which add their tiles in rank order through distributed shared memory: no workspace, one launch.
// VEC: rows of x and W allow 16-byte loads. fp32, 9728 x 896 on 600 rows: 397 us (26 TFLOP/s); with the attention of
// prefill_attention.cu, Qwen2-0.5B in fp32 on 2 x 300 tokens takes 20.9 ms (54.6 with 4 x 4 outputs a thread, unbuffered).
constexpr int kTiledThreads = 128, kTile = 64, kTileK = 16;

template <typename T, bool VEC>
__global__ void __launch_bounds__(kTiledThreads) linear_tiled_kernel(const LinearParamsGeneric<T> p) {
  constexpr int kPitch = kTile + 4;
  __shared__ __align__(16) float tiles[2][2][kTileK][kPitch];  // [buffer][x, W][k][row]: also the tile handed over
  static_assert(sizeof(tiles) >= sizeof(float) * kTile * kTile, "the tile's sums must fit the operand buffers");
  const int tx = threadIdx.x % 8, ty = threadIdx.x / 8;  // 8 columns of 8, 16 rows of 4
  const int m_base = blockIdx.y * kTile, n_base = blockIdx.x * kTile;
  const int splits = gridDim.z, blocks = (p.k + kTileK - 1) / kTileK, per = (blocks + splits - 1) / splits;
  const int first = blockIdx.z * per, last = min(first + per, blocks);

  float staged[2][8];
  auto fetch = [&](int block) {
    if constexpr (VEC) {  // two 16-byte loads of 4 k each (fp32)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = threadIdx.x / 4 + 32 * h, k = block * kTileK + threadIdx.x % 4 * 4;
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
        if (m_base + r < p.m && k < p.k)
          a = __ldg(reinterpret_cast<const float4*>(p.x + (m_base + r) * p.x_row_stride + k));
        if (n_base + r < p.n && k < p.k)
          b = __ldg(reinterpret_cast<const float4*>(p.w + static_cast<int64_t>(n_base + r) * p.k + k));
        staged[0][h * 4] = a.x; staged[0][h * 4 + 1] = a.y; staged[0][h * 4 + 2] = a.z; staged[0][h * 4 + 3] = a.w;
        staged[1][h * 4] = b.x; staged[1][h * 4 + 1] = b.y; staged[1][h * 4 + 2] = b.z; staged[1][h * 4 + 3] = b.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int id = i * kTiledThreads + threadIdx.x, r = id / kTileK, k = block * kTileK + id % kTileK;
        staged[0][i] = m_base + r < p.m && k < p.k ? Elem<T>::load(p.x + (m_base + r) * p.x_row_stride + k) : 0.0f;
        staged[1][i] = n_base + r < p.n && k < p.k ? Elem<T>::load(p.w + static_cast<int64_t>(n_base + r) * p.k + k) : 0.0f;
      }
    }
  };
  auto place = [&](int buffer) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int id = i * kTiledThreads + threadIdx.x;
      const int r = VEC ? threadIdx.x / 4 + 32 * (i / 4) : id / kTileK;
      const int k = VEC ? threadIdx.x % 4 * 4 + i % 4 : id % kTileK;
      tiles[buffer][0][k][r] = staged[0][i];
      tiles[buffer][1][k][r] = staged[1][i];
    }
  };

  float acc[4][8] = {};
  if (first < last) {
    fetch(first);
    place(0);
  }
  __syncthreads();
  for (int block = first; block < last; ++block) {
    const int buffer = (block - first) & 1;
    if (block + 1 < last) fetch(block + 1);
    float sum[4][8] = {};
#pragma unroll
    for (int k = 0; k < kTileK; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(&tiles[buffer][0][k][ty * 4]);
      const float4 b0 = *reinterpret_cast<const float4*>(&tiles[buffer][1][k][tx * 4]);
      const float4 b1 = *reinterpret_cast<const float4*>(&tiles[buffer][1][k][32 + tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[i][j] = fmaf(av[i], bv[j], sum[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] += sum[i][j];
    if (block + 1 < last) place(buffer ^ 1);
    __syncthreads();
  }
  auto column = [&](int j) { return (j >> 2) * 32 + tx * 4 + (j & 3); };
  if (splits == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        epilogue_generic(p, m_base + ty * 4 + i, n_base + column(j), acc[i][j], j < 7 ? acc[i][j + 1] : 0.0f);
    return;
  }
  float* mine = &tiles[0][0][0][0];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; j += 4)
      *reinterpret_cast<float4*>(mine + (ty * 4 + i) * kTile + column(j)) =
          make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
  cluster_sync();
  const int rank = cluster_cta_rank();
  for (int unit = rank * kTiledThreads + threadIdx.x; unit < kTile * kTile / 4; unit += splits * kTiledThreads) {
    float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int s = 0; s < splits; ++s) {
      const float4 t = load_cluster_f32x4(smem_u32(mine + unit * 4), s);
      total.x += t.x; total.y += t.y; total.z += t.z; total.w += t.w;
    }
    const int m = m_base + unit / (kTile / 4), n = n_base + unit % (kTile / 4) * 4;
    epilogue_generic(p, m, n, total.x, total.y);
    epilogue_generic(p, m, n + 1, total.y, 0.0f);
    epilogue_generic(p, m, n + 2, total.z, total.w);
    epilogue_generic(p, m, n + 3, total.w, 0.0f);
  }
  cluster_sync();  // no CTA leaves while another reads its tile
}

struct TilePlan {
  int bm, bn, threads, splits, tiles_m, tiles_n;
  int64_t partial_floats_per_tile_split;
};

TilePlan plan_warp_level(int64_t m, int64_t k, int64_t n) {
  TilePlan t;
  if (m <= 16) {
    t.bm = 16; t.bn = 64; t.threads = 128;
  } else if (m <= 32) {
    t.bm = 32; t.bn = 64; t.threads = 128;
  } else if (m <= 64) {
    t.bm = 64; t.bn = 64; t.threads = 128;
  } else {
    t.bm = 128; t.bn = 128; t.threads = 256;
  }
  t.tiles_m = static_cast<int>(ceil_div(m, t.bm));
  t.tiles_n = static_cast<int>(ceil_div(n, t.bn));
  const int64_t tiles = static_cast<int64_t>(t.tiles_m) * t.tiles_n;
  const int64_t kb = ceil_div(k, kBK);
  int64_t splits = 1;
  const int64_t target = 2 * kNumSMs;
  if (tiles < target) {
    splits = ceil_div(target, tiles);
    if (splits > 8) splits = 8;
    if (splits > kb) splits = kb;
    // no empty splits: every split gets at least one k block
    const int64_t per = ceil_div(kb, splits);
    splits = ceil_div(kb, per);
  }
  t.splits = static_cast<int>(splits);
  t.partial_floats_per_tile_split = static_cast<int64_t>(t.bm) * t.bn;
  return t;
}

// The tile counters sit in a fixed-size region at the start of the workspace, so that calls
// with different tile grids can share one workspace: the region is only ever touched as
// counters (and left at zero), never as partial sums. Split-K is used for < 2 * 148 tiles.
constexpr int64_t kCounterBytes = 4096;
int64_t counters_bytes(const TilePlan& t) {
  (void)t;
  return kCounterBytes;
}
static_assert(2 * kNumSMs * 4 <= kCounterBytes, "counter region too small");

template <int BM, int BN, int WM, int WN, int STAGES, typename T>
int launch_tile(const LinearParams<T>& p, const TilePlan& t, cudaStream_t stream) {
  constexpr int smem = STAGES * (BM + BN) * 128;
  auto kernel = linear_warp_kernel<T, BM, BN, WM, WN, STAGES>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return B200_ERR_LAUNCH;
  dim3 grid(t.tiles_n, t.tiles_m, t.splits);
  kernel<<<grid, WM * WN * 32, smem, stream>>>(p);
  return launch_status();
}

}  // namespace
}  // namespace b200

namespace b200 {
int linear_tcgen05(const void* input, const void* weight, const void* bias, const void* residual,
                   void* output, int64_t m, int64_t k, int64_t n, int64_t input_row_stride, int dtype,
                   int epilogue, int32_t* status, cudaStream_t stream, bool fold_norm = false,
                   double norm_eps = 0.0, const float* norm_squares = nullptr, int norm_slices = 0);
}

using namespace b200;

// The tcgen05 path takes every problem it can fill the GPU with (it declines decode-size M
// with few N tiles, which need split-K); B200_LINEAR_PATH=mma.sync or the launch-mode flag
// B200_LAUNCH_LINEAR_WARP_LEVEL (what a dispatch plan sets) force the warp-level kernel.
static bool use_tcgen05(int64_t m) {
  (void)m;
  if ((launch_mode() & B200_LAUNCH_LINEAR_WARP_LEVEL) != 0) return false;
  const char* value = getenv("B200_LINEAR_PATH");
  return value == nullptr || strcmp(value, "mma.sync") != 0;
}

extern "C" int64_t b200_linear_workspace_bytes(int64_t m, int64_t k, int64_t n, int dtype,
                                               int epilogue) {
  (void)epilogue;
  if ((dtype != B200_BF16 && dtype != B200_F16) || m <= 0 || k <= 0 || n <= 0) return 0;
  const TilePlan t = plan_warp_level(m, k, n);
  if (t.splits <= 1) return 0;
  return counters_bytes(t) + static_cast<int64_t>(t.tiles_m) * t.tiles_n * t.splits *
                                 t.partial_floats_per_tile_split * 4;
}

// Rows up to which W is streamed (linear_rows_kernel, whose time grows with every 8 rows) instead of multiplied in tiles
// (the same time for 1 to 64 rows). 8, 16, 32, 40 rows against tiles, us in a chain of launches: 9728 x 896 12.0, 18.6,
// 33.6, 41.3 against 58; 896 x 4864 7.8, 14.5, 24.8, 25.6 against 45. Matrices beyond L2, which every 8 rows read again:
// 37888 x 3584 126, 246, 473, 590 against 856; 3584 x 18944 79, 144, 247, 298 against 576; LM head 151936 x 896 125, 244,
// 479, 597 against 646.
constexpr int64_t kRowsLimit = 40;
// A short K leaves most of a CTA's 4 x 128 k idle, so that every 8 rows more cost as much as with a long one, while tiles
// cost in proportion to K. 12000 columns, K 128, 384, 768: 16 rows 13.0, 15.5, 21.0 us against 13.5, 24.7, 44.2 in tiles,
// 24 rows 18.1, 22.0, 30.2 against 14.0, 25.1, 44.9, 40 rows 28.3, 34.5, 46.9 against 14.1, 25.9, 45.7. As long as the
// CTAs are few (1024 columns, 40 rows, K 128: 5.3 against 10.4; 4096 columns, 24 rows, K 128: 7.9 against 10.3) this
// does not show.
static bool streams_rows(int64_t m, int64_t k, int64_t n) {
  const int64_t tall = ceil_div(m, static_cast<int64_t>(kRowsOfX));
  return m <= kRowsLimit && (tall == 1 || ceil_div(n, static_cast<int64_t>(kRowsColumns)) * tall <= 16 * kNumSMs ||
                             k >= 192 * (tall - 1));
}

// How a streamed projection is cut: groups of columns x row tiles x CTAs of a cluster along K, and the stages of a ring.
struct RowsGrid {
  int64_t groups, tall, splits;
  int slots;
};
static RowsGrid rows_grid(int rows, int64_t m, int64_t k, int64_t n) {
  // with few columns as many CTAs of a cluster along K as it takes to hold W in one ring each, up to some eight an SM
  const int64_t groups = ceil_div(n, kRowsColumns), tall = ceil_div(m, static_cast<int64_t>(rows)), chunks = ceil_div(k, kRowsChunk);
  int64_t splits = ceil_div(chunks, kRowsWarps * kRowsRing);
  if (splits > 8 * kNumSMs / (groups * tall)) splits = 8 * kNumSMs / (groups * tall);
  if (splits > 8) splits = 8;
  if (splits < 1) splits = 1;
  const int64_t most = ceil_div(chunks, kRowsWarps * splits);
  return RowsGrid{groups, tall, splits, static_cast<int>(most < kRowsRing ? most : kRowsRing)};
}

// Whether the norm belongs inside: that saves a launch, but every CTA squares and scales x beside its products (a quarter
// more arithmetic) and holds more registers, so that an SM may hold fewer. It pays while both forms take one wave of CTAs
// (240 random sizes in chains of launches: 0.61 to 0.91 of the two launches), and mostly with two waves each (0.75 to 1.06;
// 4 rows with full rings excepted: 0.99 to 1.09). Beyond, or where the norm adds a wave, it loses: 32 rows, 2560 x 454
// 8.6 -> 11.8 us, 9 rows, 512 x 23918 31 -> 38, 1 row, 4096 x 14648 44 -> 58. Decode steps, two launches -> one everywhere
// -> by this rule: 24 layers of Qwen2-0.5B, 4 sequences 980 -> 944 -> 943 us, 32 sequences 2938 -> 3159 -> 2944; 4 layers
// of Qwen2-7B, 1 sequence 853 -> 1005 -> 847.
static bool norm_pays_inside(int64_t m, int64_t k, int64_t n) {
  const int rows = m <= 4 ? 4 : 8;
  const RowsGrid g = rows_grid(rows, m, k, n);
  auto waves = [&](int64_t registers) {
    const int64_t by_registers = 64 * 1024 / (registers * kRowsThreads);
    const int64_t by_memory = 227 * 1024 / (kRowsWarps * g.slots * kRowsChunkBytes + 3 * 1024);
    return ceil_div(g.groups * g.tall * g.splits, kNumSMs * (by_registers < by_memory ? by_registers : by_memory));
  };
  // registers of a thread as the compiler reports them: linear_rows_kernel<4> 80, with the norm 96; <8> 128 and 168
  const int64_t with = waves(rows == 4 ? 96 : 168), without = waves(rows == 4 ? 80 : 128);
  return with == without && (with == 1 || (with == 2 && (rows == 8 || g.slots < kRowsRing)));
}

template <int ROWS, bool NORM>
static int launch_rows_of(const LinearParamsGeneric<float>& p, cudaStream_t s) {
  const RowsGrid g = rows_grid(ROWS, p.m, p.k, p.n);
  const int smem = kRowsWarps * g.slots * kRowsChunkBytes;
  if (cudaFuncSetAttribute((linear_rows_kernel<ROWS, NORM>), cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kRowsWarps * kRowsRing * kRowsChunkBytes) != cudaSuccess)
    return B200_ERR_LAUNCH;
  const dim3 grid(static_cast<unsigned>(g.groups), static_cast<unsigned>(g.tall), static_cast<unsigned>(g.splits));
  const int early = (launch_mode() & B200_LAUNCH_CONSTANT_WEIGHTS) != 0 ? 1 : 0;
  return launch_chained_cluster_xz(linear_rows_kernel<ROWS, NORM>, grid, dim3(kRowsThreads), static_cast<size_t>(smem), s, 1u,
                                   static_cast<unsigned>(g.splits), p, g.slots, early) == cudaSuccess
             ? launch_status() : B200_ERR_LAUNCH;
}
template <bool NORM>
static int launch_rows(const LinearParamsGeneric<float>& p, cudaStream_t s) {
  return p.m <= 4 ? launch_rows_of<4, NORM>(p, s) : launch_rows_of<8, NORM>(p, s);
}

template <typename T>
static int linear_generic(const void* input, const void* weight, const void* bias, const void* residual, void* output,
                          int64_t m, int64_t k, int64_t n, int64_t input_row_stride, int epilogue, cudaStream_t s) {
  LinearParamsGeneric<T> p;
  p.x = static_cast<const T*>(input);
  p.w = static_cast<const T*>(weight);
  p.bias = static_cast<const T*>(bias);
  p.residual = static_cast<const T*>(residual);
  p.out = static_cast<T*>(output);
  p.x_row_stride = input_row_stride;
  p.m = static_cast<int>(m);
  p.k = static_cast<int>(k);
  p.n = static_cast<int>(n);
  p.epilogue = epilogue;
  bool vec = false;
  if constexpr (sizeof(T) == 4) {
    vec = k % 4 == 0 && input_row_stride % 4 == 0 && aligned16(input) && aligned16(weight);
    if (vec && streams_rows(m, k, n)) return launch_rows<false>(p, s);
  }
  const int64_t tiles_m = ceil_div(m, kTile), tiles_n = ceil_div(n, kTile);
  if (tiles_m > 65535) return B200_ERR_TOO_LARGE;
  // CTAs of a tile: as many K slices (of at least 8 blocks) as bring some 4 CTAs to every SM
  int64_t splits = 1;
  while (splits < 8 && tiles_m * tiles_n * splits * 2 <= 4 * kNumSMs && ceil_div(k, kTileK) >= 16 * splits) splits *= 2;
  dim3 grid(static_cast<unsigned>(tiles_n), static_cast<unsigned>(tiles_m), static_cast<unsigned>(splits));
  auto launch_with = [&](auto kernel) {
    if (splits == 1) kernel<<<grid, kTiledThreads, 0, s>>>(p);
    else if (launch_cluster_z(kernel, grid, kTiledThreads, s, static_cast<unsigned>(splits), p) != cudaSuccess)
      return B200_ERR_LAUNCH;
    return launch_status();
  };
  if constexpr (sizeof(T) == 4) {
    if (vec) return launch_with(linear_tiled_kernel<T, true>);
  }
  return launch_with(linear_tiled_kernel<T, false>);
}

// The tensor-core kernels, bf16 or fp16 (T): tcgen05, or the warp-level kernel where that declines.
template <typename T>
static int linear_tensor_core(const void* input, const void* weight, const void* bias, const void* residual,
                              void* output, int64_t m, int64_t k, int64_t n, int64_t input_row_stride, int dtype,
                              int epilogue, void* workspace, int64_t workspace_bytes, int32_t* status,
                              cudaStream_t s) {
  if (use_tcgen05(m)) {
    const int code = linear_tcgen05(input, weight, bias, residual, output, m, k, n, input_row_stride, dtype,
                                    epilogue, status, s);
    if (code != B200_ERR_UNSUPPORTED) return code;
  }
  const TilePlan t = plan_warp_level(m, k, n);
  if (t.tiles_m > 65535) return B200_ERR_TOO_LARGE;
  LinearParams<T> p;
  p.x = static_cast<const T*>(input);
  p.w = static_cast<const T*>(weight);
  p.bias = static_cast<const T*>(bias);
  p.residual = static_cast<const T*>(residual);
  p.out = static_cast<T*>(output);
  p.x_row_stride = input_row_stride;
  p.m = static_cast<int>(m);
  p.k = static_cast<int>(k);
  p.n = static_cast<int>(n);
  p.splits = t.splits;
  p.epilogue = epilogue;
  p.partials = nullptr;
  p.counters = nullptr;
  if (t.splits > 1) {
    const int64_t need = b200_linear_workspace_bytes(m, k, n, dtype, epilogue);
    if (!workspace || workspace_bytes < need) return B200_ERR_WORKSPACE;
    p.counters = static_cast<int*>(workspace);
    p.partials = reinterpret_cast<float*>(static_cast<char*>(workspace) + counters_bytes(t));
  }
  if (t.bm == 16) return launch_tile<16, 64, 1, 4, 4>(p, t, s);
  if (t.bm == 32) return launch_tile<32, 64, 1, 4, 4>(p, t, s);
  if (t.bm == 64) return launch_tile<64, 64, 1, 4, 4>(p, t, s);
  return launch_tile<128, 128, 2, 4, 3>(p, t, s);
}

extern "C" int b200_linear(const void* input, const void* weight, const void* bias,
                           const void* residual, void* output, int64_t m, int64_t k, int64_t n,
                           int64_t input_row_stride, int dtype, int epilogue, void* workspace,
                           int64_t workspace_bytes, int32_t* status, void* stream) {
  if (!input || !weight || !output || m < 0 || k <= 0 || n <= 0 || input_row_stride < k)
    return B200_ERR_BAD_ARGUMENT;
  if (epilogue != B200_EPILOGUE_NONE && epilogue != B200_EPILOGUE_RESIDUAL &&
      epilogue != B200_EPILOGUE_SWIGLU)
    return B200_ERR_BAD_ARGUMENT;
  if (epilogue == B200_EPILOGUE_RESIDUAL && !residual) return B200_ERR_BAD_ARGUMENT;
  if (epilogue == B200_EPILOGUE_SWIGLU && n % 2 != 0) return B200_ERR_BAD_ARGUMENT;
  if (m == 0) return B200_OK;
  if (m > INT32_MAX || k > INT32_MAX || n > INT32_MAX) return B200_ERR_TOO_LARGE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);

  if (dtype == B200_F32)
    return linear_generic<float>(input, weight, bias, residual, output, m, k, n, input_row_stride, epilogue, s);
  if (dtype == B200_F16) {
    // fp16 on the tensor cores where 16-byte copies reach every row (the four projections of a Qwen2-0.5B layer on
    // 1030 rows: 478 us each on average on the CUDA cores, 21.6 us here); what they do not reach (and a caller
    // without the workspace that split K needs) keeps the CUDA-core kernel
    const int64_t need = b200_linear_workspace_bytes(m, k, n, dtype, epilogue);
    if (k % 8 != 0 || input_row_stride % 8 != 0 || !aligned16(input) || !aligned16(weight) ||
        (need > 0 && (!workspace || workspace_bytes < need)))
      return linear_generic<__half>(input, weight, bias, residual, output, m, k, n, input_row_stride, epilogue, s);
    return linear_tensor_core<__half>(input, weight, bias, residual, output, m, k, n, input_row_stride, dtype,
                                      epilogue, workspace, workspace_bytes, status, s);
  }
  if (dtype != B200_BF16) return B200_ERR_UNSUPPORTED;
  if (k % 8 != 0 || input_row_stride % 8 != 0) return B200_ERR_UNSUPPORTED;
  if (!aligned16(input) || !aligned16(weight)) return B200_ERR_ALIGNMENT;
  return linear_tensor_core<__nv_bfloat16>(input, weight, bias, residual, output, m, k, n, input_row_stride, dtype,
                                           epilogue, workspace, workspace_bytes, status, s);
}

extern "C" int b200_rms_norm_linear_pays(int64_t m, int64_t k, int64_t n) {
  return m > 0 && k > 0 && n > 0 && streams_rows(m, k, n) && norm_pays_inside(m, k, n) ? 1 : 0;
}

extern "C" int b200_rms_norm_linear(const void* input, const void* norm_weight, const void* weight, const void* bias,
                                    void* output, int64_t m, int64_t k, int64_t n, int64_t input_row_stride,
                                    double epsilon, int dtype, int epilogue, void* stream) {
  if (!input || !norm_weight || !weight || !output || m < 0 || k <= 0 || n <= 0 || input_row_stride < k || !(epsilon >= 0.0))
    return B200_ERR_BAD_ARGUMENT;
  if (epilogue != B200_EPILOGUE_NONE && epilogue != B200_EPILOGUE_SWIGLU) return B200_ERR_BAD_ARGUMENT;
  if (epilogue == B200_EPILOGUE_SWIGLU && n % 2 != 0) return B200_ERR_BAD_ARGUMENT;
  if (m == 0) return B200_OK;
  if (m > INT32_MAX || k > INT32_MAX || n > INT32_MAX) return B200_ERR_TOO_LARGE;
  if (dtype != B200_F32 || k % 4 != 0 || input_row_stride % 4 != 0 || !aligned16(input) || !aligned16(norm_weight) ||
      !aligned16(weight) || !streams_rows(m, k, n))
    return B200_ERR_UNSUPPORTED;
  LinearParamsGeneric<float> p;
  p.x = static_cast<const float*>(input);
  p.w = static_cast<const float*>(weight);
  p.bias = static_cast<const float*>(bias);
  p.residual = nullptr;
  p.out = static_cast<float*>(output);
  p.x_row_stride = input_row_stride;
  p.m = static_cast<int>(m);
  p.k = static_cast<int>(k);
  p.n = static_cast<int>(n);
  p.epilogue = epilogue;
  p.norm_weight = static_cast<const float*>(norm_weight);
  p.norm_eps = static_cast<float>(epsilon);
  return launch_rows<true>(p, static_cast<cudaStream_t>(stream));
}
