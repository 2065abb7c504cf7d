// Projections of a few rows (one conversation, a small batch) in 16-bit types: y[M,N] = x[M,K] W[N,K]^T with M up to
// 8, in every form that a decode step has: plain with bias / residual / SwiGLU, fp32 sums for the operator behind it,
// folded RMSNorm.
//
// Bound by reading W once and, in a 0.5B model (2 - 17 MB a launch), by the chain launch -> x -> product -> sum ->
// store. So W travels as early as it can, before the dependency wait, and what is behind the wait is short: one read
// of x, a handful of warp-level products, one exchange between the warps and the store. Every warp has a K range of
// its own and every lane a ring of 16-byte pieces that it alone fills (cp.async) and reads: shared memory as more
// registers, so that the next launch's W finds room while this one is at work, and no barrier in the main loop. The
// rows of W are the M side of m16n8k16 and the rows of x its N side. The order of k inside a product is free as long
// as both operands share it: a lane takes 8 neighbouring k of its W rows and of its x row, the first half as one
// product's fragment, the second half as the next one's.
//
// Qwen2-0.5B on 1 row, launches in a chain, against the tcgen05 kernels (whose prologue, ring of tiles, tensor memory and
// cluster exchange cost 3.7 us however small the matrix): q|k|v 3.7 -> 2.3 us, o 4.9 -> 2.5, gate|up 10.1 -> 4.7
// (17.4 MB, 3.7 TB/s), down 7.2 -> 4.5, LM head 56 -> 55; 8 rows within 15 % of that. Decode step 935 -> 648 us (8
// rows: 913 -> 688), four layers of the 7B 692 -> 628 (693 -> 667), Bazirax 1.5b 546 -> 431 (563 -> 454), Lozanex 1.5b
// 511 -> 465 (745 -> 712).
#include <stdlib.h>

#include "common.cuh"
#include "linear_rows.cuh"

namespace b200 {
namespace {

constexpr int kChunk = 32;   // k of two products: 4 lanes x 8
constexpr int kHalf = 4;     // chunks of half a ring: a copy group
constexpr int kRows = 8;     // rows of x, the N side of a product
constexpr int kColumns = 16; // columns of y of a CTA, the M side
constexpr int kPieces = 2;   // 16-byte pieces of W of a lane and chunk
constexpr int kWarps = 4, kThreads = kWarps * 32;

template <typename T>
struct RowsParams {
  const T* x;
  const T* w;
  const T* bias;
  const T* residual;
  T* out;
  float* sums;         // fp32 sums instead of `out`
  float* row_squares;  // and sum(x_r^2), written by the first CTA
  int64_t x_row_stride;
  int m, k, n, epilogue;
  int fold_norm;
  float norm_eps;
  int slots;  // chunks that a warp's ring has room for: 2 kHalf, or all that it has to multiply if fewer
  int early;  // W may be read before the kernels in front have finished
};

// x by way of L1: all CTAs of an SM read the same few kilobytes, whose L2 slices would otherwise answer each of them
// (gate|up on 8 rows: 6.5 us past L1, 5.3 us through it)
__device__ __forceinline__ uint4 load_rows_of_x(const void* p) {
  uint4 v;
  asm volatile("ld.global.ca.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

// as in the tcgen05 projections: a few ulp of fp32, far below the rounding that follows
__device__ __forceinline__ float silu_fast(float x) { return __fdividef(x, 1.0f + exp2f(-1.4426950408889634f * x)); }

template <typename T>
__device__ __forceinline__ float square_pair(uint32_t pair, float sum) {
  const float a = Elem<T>::lo(pair), b = Elem<T>::hi(pair);
  return fmaf(b, b, fmaf(a, a, sum));
}

template <typename T, bool SQUARES>
__global__ void __launch_bounds__(kThreads) linear_rows16_kernel(const RowsParams<T> p) {
  constexpr int kPitch = kColumns + 4;  // conflict-free fragment stores
  extern __shared__ __align__(16) unsigned char ring[];  // [warp][chunk][piece][lane]
  __shared__ __align__(16) float part[kWarps][kRows][kPitch];
  __shared__ float total[kRows][kColumns];
  __shared__ float squares[kWarps][kRows];
  __shared__ float total_squares[kRows];
  grid_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * kColumns, splits = gridDim.z, rank = blockIdx.z;
  const int chunks = (p.k + kChunk - 1) / kChunk, parts = splits * kWarps, mine = rank * kWarps + warp;
  const int first = static_cast<int>(static_cast<int64_t>(chunks) * mine / parts);
  const int count = static_cast<int>(static_cast<int64_t>(chunks) * (mine + 1) / parts) - first;
  const uint32_t base = smem_u32(ring) + warp * (p.slots * kPieces * 512) + lane * 16;

  // Chunk c of this warp goes to slot c % (2 kHalf). (Pieces beyond K become zeros; columns beyond N are not copied:
  // what they multiply is not stored.)
  auto copy_weights = [&](int c) {
    if (c >= count) return;
    const int k = (first + c) * kChunk + t * 8;
    const bool there = k < p.k;  // (K is a multiple of 8: all 8 or none)
    const uint32_t at = base + c % (2 * kHalf) * (kPieces * 512);
#pragma unroll
    for (int r = 0; r < kPieces; ++r) {
      const int n = n0 + r * 8 + g;
      if (n < p.n) cp_async16_zfill(at + r * 512, p.w + static_cast<int64_t>(n) * p.k + (there ? k : 0), there ? 16 : 0);
    }
  };
  // x is read into registers, all of it that the ring covers at once
  uint4 xv[2 * kHalf];
  const T* x_row = p.x + (g < p.m ? g : 0) * p.x_row_stride + t * 8;
  auto load_row = [&](int slot, int c) {
    const int k = (first + c) * kChunk;
    xv[slot] = make_uint4(0u, 0u, 0u, 0u);
    if (g < p.m && c < count && k + t * 8 < p.k) xv[slot] = load_rows_of_x(x_row + k);
  };
  if (!p.early) grid_dependency_wait();
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // two copy groups in flight
#pragma unroll
    for (int j = 0; j < kHalf; ++j) copy_weights(h * kHalf + j);
    cp_async_commit();
  }
  if (p.early) grid_dependency_wait();
#pragma unroll
  for (int c = 0; c < 2 * kHalf; ++c) load_row(c, c);

  float acc[2][4] = {};  // (two chains of products, added at the end)
  float ss = 0.0f;
  for (int turn = 0; turn < count; turn += 2 * kHalf) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c0 = turn + h * kHalf;
      if (c0 >= count) break;
      cp_async_wait<1>();
      uint4 v[kHalf][kPieces];
#pragma unroll
      for (int j = 0; j < kHalf; ++j)
#pragma unroll
        for (int r = 0; r < kPieces; ++r)
          if (c0 + j < count)
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(v[j][r].x), "=r"(v[j][r].y), "=r"(v[j][r].z), "=r"(v[j][r].w)
                         : "r"(base + (h * kHalf + j) * (kPieces * 512) + r * 512) : "memory");
#pragma unroll
      for (int j = 0; j < kHalf; ++j) {
        if (c0 + j >= count) break;
        const uint4 b = xv[h * kHalf + j], u = v[j][0], d = v[j][1];
        const uint32_t low[4] = {u.x, d.x, u.y, d.y}, high[4] = {u.z, d.z, u.w, d.w};
        mma_16816<T>(acc[0], low, b.x, b.y);
        mma_16816<T>(acc[1], high, b.z, b.w);
        if (SQUARES) ss = square_pair<T>(b.w, square_pair<T>(b.z, square_pair<T>(b.y, square_pair<T>(b.x, ss))));
      }
#pragma unroll
      for (int j = 0; j < kHalf; ++j) {  // (every lane refills the pieces that it has read itself)
        copy_weights(c0 + 2 * kHalf + j);
        load_row(h * kHalf + j, c0 + 2 * kHalf + j);
      }
      cp_async_commit();
    }
  }
  cp_async_wait<0>();

  // the warps' sums, in warp order (behind them, with several CTAs, in rank order: the same result every time)
  float* at = &part[warp][2 * t][g];
  at[0] = acc[0][0] + acc[1][0];
  at[kPitch] = acc[0][1] + acc[1][1];
  at[8] = acc[0][2] + acc[1][2];
  at[kPitch + 8] = acc[0][3] + acc[1][3];
  if (SQUARES) {
    ss += __shfl_xor_sync(0xffffffffu, ss, 1);
    ss += __shfl_xor_sync(0xffffffffu, ss, 2);
    if (t == 0) squares[warp][g] = ss;
  }
  __syncthreads();
  if (splits > 1) {
    for (int u = threadIdx.x; u < kRows * kColumns; u += kThreads) {
      float sum = 0.0f;
#pragma unroll
      for (int s = 0; s < kWarps; ++s) sum += part[s][u / kColumns][u % kColumns];
      total[u / kColumns][u % kColumns] = sum;
    }
    if (SQUARES && threadIdx.x < kRows) {
      float sum = 0.0f;
#pragma unroll
      for (int s = 0; s < kWarps; ++s) sum += squares[s][threadIdx.x];
      total_squares[threadIdx.x] = sum;
    }
    cluster_sync();
  }
  // pairs of neighbouring columns, dealt to the CTAs of the cluster
  for (int u = rank + splits * threadIdx.x; u < kRows * kColumns / 2; u += splits * kThreads) {
    const int row = u / (kColumns / 2), c = u % (kColumns / 2) * 2, n = n0 + c;
    if (row >= p.m || n >= p.n) continue;
    const bool has1 = n + 1 < p.n;
    float v0 = 0.0f, v1 = 0.0f, sq = 0.0f;
    if (splits > 1) {
      for (int s = 0; s < splits; ++s) {
        v0 += load_cluster_f32(smem_u32(&total[row][c]), s);
        v1 += load_cluster_f32(smem_u32(&total[row][c + 1]), s);
        if (SQUARES) sq += load_cluster_f32(smem_u32(&total_squares[row]), s);
      }
    } else {
#pragma unroll
      for (int s = 0; s < kWarps; ++s) {
        const float2 v = *reinterpret_cast<const float2*>(&part[s][row][c]);
        v0 += v.x;
        v1 += v.y;
        if (SQUARES) sq += squares[s][row];
      }
    }
    const int64_t o = static_cast<int64_t>(row) * p.n + n;
    if (p.sums != nullptr) {
      p.sums[o] = v0;
      if (has1) p.sums[o + 1] = v1;
      if (SQUARES && n == 0 && p.row_squares != nullptr) p.row_squares[row] = sq;
      continue;
    }
    if (SQUARES && p.fold_norm) {
      const float scale = rsqrtf(sq / static_cast<float>(p.k) + p.norm_eps);
      v0 *= scale;
      v1 *= scale;
    }
    if (p.bias != nullptr) {
      v0 += Elem<T>::load(p.bias + n);
      if (has1) v1 += Elem<T>::load(p.bias + n + 1);
    }
    Elem<T>::round_pair(v0, v1);
    if (p.epilogue == B200_EPILOGUE_SWIGLU) {  // column 2j is gate_j, column 2j + 1 is up_j
      Elem<T>::store(p.out + static_cast<int64_t>(row) * (p.n / 2) + n / 2, Elem<T>::round(silu_fast(v0)) * v1);
      continue;
    }
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
  if (splits > 1) cluster_sync();  // no CTA leaves while another reads its sums
}

template <typename T>
int linear_few_rows_of(const FewRowsCall& c, cudaStream_t stream) {
  constexpr int kSlotBytes = kWarps * kPieces * 512;
  // With few columns as many CTAs of a cluster along K as it takes to hold W in one ring each, up to some four CTAs
  // an SM (896 x 4864 on 1 row: 4.5 us with 5 CTAs a column tile; 7.2 us on the tcgen05 kernel in clusters).
  const int64_t groups = ceil_div(c.n, kColumns), chunks = ceil_div(c.k, kChunk);
  int64_t splits = ceil_div(chunks, kWarps * 2 * kHalf);
  if (splits > 4 * kNumSMs / groups) splits = 4 * kNumSMs / groups;
  if (splits > 8) splits = 8;
  if (splits < 1) splits = 1;
  const int64_t most = ceil_div(chunks, kWarps * splits);

  RowsParams<T> p;
  p.x = static_cast<const T*>(c.input);
  p.w = static_cast<const T*>(c.weight);
  p.bias = static_cast<const T*>(c.bias);
  p.residual = static_cast<const T*>(c.residual);
  p.out = static_cast<T*>(c.output);
  p.sums = c.sums;
  p.row_squares = c.row_squares;
  p.x_row_stride = c.input_row_stride;
  p.m = static_cast<int>(c.m);
  p.k = static_cast<int>(c.k);
  p.n = static_cast<int>(c.n);
  p.epilogue = c.epilogue;
  p.fold_norm = c.fold_norm ? 1 : 0;
  p.norm_eps = static_cast<float>(c.norm_eps);
  p.slots = static_cast<int>(most < 2 * kHalf ? most : 2 * kHalf);
  p.early = (launch_mode() & B200_LAUNCH_CONSTANT_WEIGHTS) != 0 ? 1 : 0;
  const bool squares = c.fold_norm || c.row_squares != nullptr;
  const dim3 grid(static_cast<unsigned>(groups), 1, static_cast<unsigned>(splits));
  auto kernel = squares ? linear_rows16_kernel<T, true> : linear_rows16_kernel<T, false>;
  if (launch_chained_cluster_xz(kernel, grid, dim3(kThreads), static_cast<size_t>(p.slots * kSlotBytes), stream, 1u,
                                static_cast<unsigned>(splits), p) != cudaSuccess)
    return B200_ERR_LAUNCH;
  return launch_status();
}

}  // namespace

// One column tile of the products: up to 8 rows it is the faster kernel at every size measured. A second one (16 rows)
// doubles what the CTAs read of x, and wins little where it wins: Qwen2-0.5B 906 -> 876 us a step, four layers of the
// 7B 696 -> 817, Lozanex 1.5b 854 -> 901.
bool takes_few_rows(int64_t m) {
  static const int64_t limit = [] {  // B200_FEW_ROWS=0: the comparison run
    const char* text = getenv("B200_FEW_ROWS");
    return text != nullptr ? static_cast<int64_t>(atoi(text)) : kRows;
  }();
  return m <= limit && m <= kRows;
}

int linear_few_rows(const FewRowsCall& call, int dtype, cudaStream_t stream) {
  return dtype == B200_F16 ? linear_few_rows_of<__half>(call, stream) : linear_few_rows_of<__nv_bfloat16>(call, stream);
}

}  // namespace b200
