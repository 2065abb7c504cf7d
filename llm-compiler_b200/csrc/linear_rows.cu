// Projections of a few rows (one conversation, a small batch) in 16-bit types: y[M,N] = x[M,K] W[N,K]^T with M up to
// 8, in every form that a decode step has: plain with bias / residual / SwiGLU, fp32 sums for the operator behind it,
// folded RMSNorm.
//
// Bound by the chain launch -> x -> product -> sum -> store: the matrices of a 0.5B model are 2 - 17 MB. The tcgen05
// kernels' prologue, ring of tiles, tensor memory and cluster exchange cost 3.7 us there however small the matrix.
// Here W travels as early as it can, before the dependency wait, and what is behind the wait is short: one read of x, a
// chain of warp-level products, one exchange and the store. A warp takes 16 columns of y (the M side of m16n8k16; the
// rows of x are its N side) and one K slice, and copies both operands into rings of its own: small CTAs with little
// shared memory, so that the next launch's W finds room while this one is at work.
//
// Qwen2-0.5B on 1 row, launches in a chain: q|k|v 3.7 -> 2.7 us, o 4.9 -> 3.6, gate|up 10.1 -> 6.9, down 7.2 -> 5.4 (8
// rows: 2.8, 3.8, 6.7, 5.5); the layer with its attention 34.3 -> 30.8 us.
//
// The sums are those of linear_tcgen05.cu bit for bit: the same K slices, each one chain of 16-deep products in K
// order, slices and squares added in the same order. (The two kinds of tensor-core instruction round alike.) So a row's
// result does not depend on how many rows stand beside it, and a token does not change with the kernel.
#include <stdlib.h>

#include "common.cuh"
#include "linear_rows.cuh"

namespace b200 {
namespace {

constexpr int kRows = 8, kColumns = 16;
constexpr int kBlock = 64;                             // k of a ring slot: 128-byte rows
constexpr int kWBytes = kColumns * 128;
constexpr int kPitch = kColumns + 4;                   // floats between rows of x in the exchange: conflict-free stores
constexpr int kPartBytes = kRows * kPitch * 4;
constexpr int kMaxSlices = 8;                          // warps of a CTA, CTAs of a cluster
constexpr int kNormFloats = 2048;                      // norm slices x rows that a CTA takes in
constexpr int kLongRing = 16, kShortRing = 4;          // slots of W of a warp
__host__ __device__ constexpr int x_ring(int ring) { return ring < 8 ? ring : 8; }  // slots of x

template <typename T>
struct RowsParams {
  const T* x;
  const T* w;
  const T* bias;
  const T* residual;
  T* out;
  float* sums;
  float* row_squares;
  float* squares_out;
  const float* norm_squares;
  int64_t x_row_stride;
  int m, k, n, epilogue;
  int splits, blocks_per_slice, warps;  // K slices, 64-k blocks of each, slices of a CTA
  int tile_groups;                      // with squares_out: 16-column groups of a tile (the cluster along x)
  int norm_slices, early;
  int slots, x_slots;  // what the rings have room for: all of a slice if it is short
  float norm_eps;
};

// x by way of L1: all CTAs of an SM read the same few kilobytes, whose L2 slices would otherwise answer each of them
__device__ __forceinline__ void copy_through_l1(uint32_t smem_addr, const void* p, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_addr), "l"(p), "r"(bytes));
}
__device__ __forceinline__ uint4 load_shared16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
template <typename T>
__device__ __forceinline__ float square_pair(uint32_t pair, float sum) {
  const float a = Elem<T>::lo(pair), b = Elem<T>::hi(pair);
  return fmaf(b, b, fmaf(a, a, sum));
}

constexpr int kPlain = 0, kSquares = 1, kNorm = 2;  // HELPER: what the warp behind the multiplying ones does

// RING: slots of a warp for blocks of W (and x_ring(RING) for blocks of x, which are near).
template <typename T, int HELPER, int RING>
__global__ void __launch_bounds__(kMaxSlices * 32) linear_rows16_kernel(const RowsParams<T> p) {
  constexpr int kXRing = x_ring(RING);
  extern __shared__ __align__(128) unsigned char ring[];  // per warp W, then per warp x, part, norm slices
  __shared__ float unit_squares[kRows][kColumns / 4];
  __shared__ float row_scale[kRows];
  grid_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * kColumns;
  const int slice = blockIdx.z * p.warps + warp;
  const int all_blocks = (p.k + kBlock - 1) / kBlock, first = slice * p.blocks_per_slice;
  const int count = warp < p.warps ? max(0, min(first + p.blocks_per_slice, all_blocks) - first) : 0;
  const int x_bytes = p.m * 128;
  const uint32_t w_base = smem_u32(ring) + warp * p.slots * kWBytes;
  const uint32_t x_base = smem_u32(ring) + p.warps * p.slots * kWBytes + warp * p.x_slots * x_bytes;
  float* parts = reinterpret_cast<float*>(ring + p.warps * (p.slots * kWBytes + p.x_slots * x_bytes));
  auto part = [&](int s, int row, int c) { return parts + (s * kRows + row) * kPitch + c; };
  float* norm_parts = parts + p.warps * kRows * kPitch;
  const bool squares = HELPER == kSquares && blockIdx.x == 0;

  // Rows of a slot are stored with their 16-byte pieces XOR-ed by the row, as a 128-byte TMA swizzle does. Pieces
  // beyond K become zeros; columns beyond N and rows beyond M are not copied: what they multiply is not stored.
  auto copy_weights = [&](int c) {
    if (c >= count) return;
    const int k = (first + c) * kBlock + (lane & 7) * 8, bytes = k < p.k ? 16 : 0;
    const uint32_t at = w_base + c % RING * kWBytes;
#pragma unroll
    for (int i = 0; i < kColumns / 4; ++i) {
      const int r = (lane >> 3) + 4 * i, n = n0 + r;
      if (n < p.n)
        cp_async16_zfill(at + r * 128 + (swizzle128(r, lane & 7) << 4), p.w + static_cast<int64_t>(n) * p.k + (bytes ? k : 0), bytes);
    }
  };
  auto copy_rows = [&](int c) {
    if (c >= count) return;
    const int k = (first + c) * kBlock + (lane & 7) * 8, bytes = k < p.k ? 16 : 0;
    const uint32_t at = x_base + c % kXRing * x_bytes;
#pragma unroll
    for (int i = 0; i < kRows / 4; ++i) {
      const int r = (lane >> 3) + 4 * i;
      if (r < p.m) copy_through_l1(at + r * 128 + (swizzle128(r, lane & 7) << 4), p.x + r * p.x_row_stride + (bytes ? k : 0), bytes);
    }
  };
  // A copy group per block of W, then one per block of x, then (in the main loop) one per turn, with the block of W
  // RING and the block of x kXRing further on. Block i is complete once group RING + i is.
  if (!p.early) grid_dependency_wait();
#pragma unroll
  for (int c = 0; c < RING; ++c) {
    copy_weights(c);
    cp_async_commit();
  }
  if (p.early) grid_dependency_wait();
#pragma unroll
  for (int c = 0; c < kXRing; ++c) {
    copy_rows(c);
    cp_async_commit();
  }
  if (squares) {  // (the whole slice stays in the ring: the helper reads x there)
    cp_async_wait<0>();
    __syncthreads();
  }

  if (warp < p.warps) {
    // fragments are read a block ahead of their products: a chain of dependent instructions has no slack for it
    struct Fragments {
      uint32_t a[4][4], b[2][4];
    } now, next;
    const int row = ((lane >> 3 & 1) << 3) + (lane & 7), x_row = min(lane & 7, p.m - 1);  // (rows beyond M: any row)
    auto read = [&](Fragments& f, int c) {
      const uint32_t w_at = w_base + c % RING * kWBytes, x_at = x_base + c % kXRing * x_bytes;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) ldmatrix_x4(f.a[ks], w_at + row * 128 + (swizzle128(row, ks * 2 + (lane >> 4)) << 4));
#pragma unroll
      for (int h = 0; h < 2; ++h) ldmatrix_x4(f.b[h], x_at + x_row * 128 + (swizzle128(x_row, h * 4 + (lane >> 3)) << 4));
    };
    float acc[4] = {};
    if (count > 0) {
      cp_async_wait<kXRing - 1>();
      __syncwarp();
      read(now, 0);
    }
    for (int c = 0; c < count; ++c) {
      if (c + 1 < count) {
        cp_async_wait<kXRing - 2>();
        __syncwarp();
        read(next, c + 1);
      }
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) mma_16816<T>(acc, now.a[ks], now.b[ks / 2][ks % 2 * 2], now.b[ks / 2][ks % 2 * 2 + 1]);
      // (every lane has read this block's slots: it did so before the barrier above)
      if (c + kXRing < count) {
        copy_weights(c + RING);
        copy_rows(c + kXRing);
      }
      cp_async_commit();
      now = next;
    }
    cp_async_wait<0>();
    float* at = part(warp, 2 * t, g);
    at[0] = acc[0];
    at[kPitch] = acc[1];
    at[8] = acc[2];
    at[kPitch + 8] = acc[3];
  } else if (HELPER == kSquares) {
    if (squares && lane < p.m) {
      const int blocks = max(0, min(static_cast<int>(blockIdx.z + 1) * p.blocks_per_slice, all_blocks) -
                                    static_cast<int>(blockIdx.z) * p.blocks_per_slice);
      const uint32_t x_row = smem_u32(ring) + p.slots * kWBytes + lane * 128;
      float ss = 0.0f;
      for (int c = 0; c < blocks; ++c) {
        uint4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = load_shared16(x_row + c * x_bytes + (((j + lane) & 7) << 4));
#pragma unroll
        for (int j = 0; j < 8; ++j)
          ss = square_pair<T>(v[j].w, square_pair<T>(v[j].z, square_pair<T>(v[j].y, square_pair<T>(v[j].x, ss))));
      }
      p.row_squares[static_cast<int64_t>(blockIdx.z) * p.m + lane] = ss;
    }
  } else if (HELPER == kNorm) {
#pragma unroll 8
    for (int i = lane; i < p.norm_slices * p.m; i += 32) norm_parts[i] = __ldcg(p.norm_squares + i);
    __syncwarp();
    if (lane < p.m) {
      float ss = 0.0f;
#pragma unroll 16
      for (int i = 0; i < p.norm_slices; ++i) ss += norm_parts[i * p.m + lane];
      row_scale[lane] = rsqrtf(ss / static_cast<float>(p.k) + p.norm_eps);
    }
  }
  __syncthreads();
  const bool across = gridDim.z > 1 && p.sums == nullptr;  // the slices are the CTAs of a cluster along z
  if (across) cluster_sync();

  // units of 4 columns, dealt to the CTAs that hold the slices
  const int owners = across ? p.splits : 1, owner = across ? blockIdx.z : 0;
  for (int u = owner + owners * threadIdx.x; u < kRows * kColumns / 4; u += owners * blockDim.x) {
    const int row = u / (kColumns / 4), c = u % (kColumns / 4) * 4, n = n0 + c, have = min(4, p.n - n);
    if (p.squares_out != nullptr) unit_squares[row][c / 4] = 0.0f;
    if (row >= p.m || have <= 0) continue;
    float v[4] = {};
    if (p.sums != nullptr) {
      float* dst = p.sums + (static_cast<int64_t>(blockIdx.z) * p.m + row) * p.n + n;
      for (int e = 0; e < have; ++e) dst[e] = *part(0, row, c + e);
      continue;
    }
    for (int s = 0; s < p.splits; ++s) {
      const uint32_t at = smem_u32(part(across ? 0 : s, row, c));
      const float4 q = across ? load_cluster_f32x4(at, s) : *reinterpret_cast<const float4*>(part(s, row, c));
      v[0] += q.x; v[1] += q.y; v[2] += q.z; v[3] += q.w;
    }
    if (HELPER == kNorm) {
      const float scale = row_scale[row];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] *= scale;
    }
    if (p.bias != nullptr) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < have) v[e] += Elem<T>::load(p.bias + n + e);
    }
    if (p.epilogue == B200_EPILOGUE_SWIGLU) {  // column 2j is gate_j, column 2j + 1 is up_j (N is even)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        if (e >= have) break;
        Elem<T>::round_pair(v[e], v[e + 1]);
        Elem<T>::store(p.out + static_cast<int64_t>(row) * (p.n / 2) + (n + e) / 2, Elem<T>::round(silu_epilogue<T>(v[e])) * v[e + 1]);
      }
      continue;
    }
    const int64_t o = static_cast<int64_t>(row) * p.n + n;
    if (p.epilogue == B200_EPILOGUE_RESIDUAL) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < have) v[e] = __fadd_rn(Elem<T>::round(v[e]), Elem<T>::load(p.residual + o + e));
    }
    if (have == 4 && (reinterpret_cast<uintptr_t>(p.out + o) & 7u) == 0) {
      *reinterpret_cast<uint2*>(p.out + o) = make_uint2(Elem<T>::pack(v[0], v[1]), Elem<T>::pack(v[2], v[3]));
    } else {
      for (int e = 0; e < have; ++e) Elem<T>::store(p.out + o + e, v[e]);
    }
    if (p.squares_out != nullptr) {  // of what was stored (here N is a multiple of 4)
      Elem<T>::round_pair(v[0], v[1]);
      Elem<T>::round_pair(v[2], v[3]);
      unit_squares[row][c / 4] = fmaf(v[0], v[0], fmaf(v[1], v[1], fmaf(v[2], v[2], v[3] * v[3])));
    }
  }
  if (p.squares_out != nullptr) {
    // unit i of a tile's rows (counted through the rows) belongs to slice i % splits, which adds its own in order
    cluster_sync();
    const int tile = blockIdx.x / p.tile_groups, member = blockIdx.x % p.tile_groups;
    for (int item = threadIdx.x * p.tile_groups + member; item < p.splits * p.m; item += blockDim.x * p.tile_groups) {
      const int s = item / p.m, row = item % p.m, units = p.tile_groups * (kColumns / 4), begin = row * units;
      float ss = 0.0f;
      for (int i = begin + (s - begin % p.splits + p.splits) % p.splits; i < begin + units; i += p.splits)
        ss += load_cluster_f32(smem_u32(&unit_squares[row][(i - begin) % 4]), (i - begin) / 4);
      p.squares_out[static_cast<int64_t>(tile * p.splits + s) * p.m + row] = ss;
    }
  }
  if (across || p.squares_out != nullptr) cluster_sync();  // no CTA leaves while another reads its part
}

template <typename T, int HELPER, int RING>
int launch_rows16(const RowsParams<T>& p, dim3 grid, int threads, unsigned cluster_x, unsigned cluster_z, cudaStream_t s) {
  auto kernel = linear_rows16_kernel<T, HELPER, RING>;
  constexpr int kMost = (RING == kShortRing ? kMaxSlices : 1) * (RING * kWBytes + x_ring(RING) * kRows * 128 + kPartBytes) +
                        (HELPER == kNorm ? kNormFloats * 4 : 0);
  const int smem = p.warps * (p.slots * kWBytes + p.x_slots * p.m * 128 + kPartBytes) +
                   (HELPER == kNorm ? p.norm_slices * p.m * 4 : 0);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost) != cudaSuccess ||
      launch_chained_cluster_xz(kernel, grid, dim3(threads), static_cast<size_t>(smem), s, cluster_x, cluster_z, p) !=
          cudaSuccess)
    return B200_ERR_LAUNCH;
  return launch_status();
}

int64_t blocks_per_slice(const FewRowsCall& c) { return ceil_div(ceil_div(c.k, kBlock), static_cast<int64_t>(c.splits)); }

template <typename T>
int linear_few_rows_of(const FewRowsCall& c, cudaStream_t stream) {
  const int64_t per = blocks_per_slice(c);
  const bool tiles = c.squares_out != nullptr;  // all slices in a CTA, the CTAs of a tile in a cluster
  const int ring = tiles ? kShortRing : kLongRing;
  RowsParams<T> p;
  p.x = static_cast<const T*>(c.input);
  p.w = static_cast<const T*>(c.weight);
  p.bias = static_cast<const T*>(c.bias);
  p.residual = static_cast<const T*>(c.residual);
  p.out = static_cast<T*>(c.output);
  p.sums = c.sums;
  p.row_squares = c.row_squares;
  p.squares_out = c.squares_out;
  p.norm_squares = c.norm_squares;
  p.x_row_stride = c.input_row_stride;
  p.m = static_cast<int>(c.m);
  p.k = static_cast<int>(c.k);
  p.n = static_cast<int>(c.n);
  p.epilogue = c.epilogue;
  p.splits = c.splits;
  p.blocks_per_slice = static_cast<int>(per);
  p.warps = tiles ? c.splits : 1;
  p.tile_groups = tiles ? c.tile_columns / kColumns : 1;
  p.norm_slices = c.norm_slices;
  p.slots = static_cast<int>(per < ring ? per : ring);
  p.x_slots = p.slots < x_ring(ring) ? p.slots : x_ring(ring);
  p.early = (launch_mode() & B200_LAUNCH_CONSTANT_WEIGHTS) != 0 ? 1 : 0;
  p.norm_eps = static_cast<float>(c.norm_eps);
  int64_t groups = ceil_div(c.n, kColumns);
  if (tiles) {
    groups = ceil_div(c.n, static_cast<int64_t>(c.tile_columns)) * p.tile_groups;
    return launch_rows16<T, kPlain, kShortRing>(p, dim3(static_cast<unsigned>(groups)), 32 * c.splits,
                                                static_cast<unsigned>(p.tile_groups), 1u, stream);
  }
  const dim3 grid(static_cast<unsigned>(groups), 1, static_cast<unsigned>(c.splits));
  if (c.row_squares != nullptr) return launch_rows16<T, kSquares, kLongRing>(p, grid, 64, 1u, 1u, stream);
  if (c.norm_squares != nullptr) return launch_rows16<T, kNorm, kLongRing>(p, grid, 64, 1u, 1u, stream);
  return launch_rows16<T, kPlain, kLongRing>(p, grid, 32, 1u, c.sums != nullptr ? 1u : static_cast<unsigned>(c.splits), stream);
}

}  // namespace

bool takes_few_rows(const FewRowsCall& c) {
  static const int64_t limit = [] {  // B200_FEW_ROWS=0: the comparison run
    const char* text = getenv("B200_FEW_ROWS");
    return text != nullptr ? static_cast<int64_t>(atoi(text)) : kRows;
  }();
  if (c.m > limit || c.m > kRows || c.splits < 1) return false;
  // A launch that is a chain of latencies. A larger matrix is a stream, which the tcgen05 kernels' TMA rings keep fuller
  // than one warp a slice can: 151936 x 896 56 against 82 us on 1 row, four layers of Qwen2-7B 688 against 955. The line
  // lies where the first form loses. us in a chain of launches, tcgen05 -> here, 1 and 8 rows, N x K in Mi elements:
  //    2.2, 1536 x 1536:   residual 6.3, 6.3 -> 4.3, 4.6; fp32 sums 3.7, 3.9 -> 2.9, 3.1; norm + SwiGLU 10.4 -> 7.2, 7.4
  //    9.0, 3072 x 3072:   residual 9.4, 9.6 -> 6.7, 8.1; fp32 sums 6.5, 6.6 -> 6.2, 5.6; norm + SwiGLU 20.6, 18.9 -> 15.1
  //    9.0, 6144 x 1536:   residual 12.1, 12.2 -> 7.9, 8.9; fp32 sums 6.8, 6.8 -> 6.2, 5.6
  //   10.0, 10240 x 1024:  residual 10.4, 10.6 -> 6.8, 7.1; fp32 sums 7.3, 7.2 -> 6.4, 8.6; norm + SwiGLU 11.2 -> 12.9 (8 rows)
  //   12.3, 3584 x 3584:   residual 11.7, 11.7 -> 8.3, 13.9
  if (c.n * c.k > (9 << 20)) return false;
  if (c.sums == nullptr && c.splits > kMaxSlices) return false;
  if (c.row_squares != nullptr && blocks_per_slice(c) > x_ring(kLongRing)) return false;  // the helper reads the whole slice
  if (c.squares_out != nullptr && c.tile_columns > kColumns * kMaxSlices) return false;
  if (c.norm_squares != nullptr && (c.splits != 1 || c.norm_slices * c.m > kNormFloats)) return false;
  return true;
}

int linear_few_rows(const FewRowsCall& call, int dtype, cudaStream_t stream) {
  return dtype == B200_F16 ? linear_few_rows_of<__half>(call, stream) : linear_few_rows_of<__nv_bfloat16>(call, stream);
}

}  // namespace b200
