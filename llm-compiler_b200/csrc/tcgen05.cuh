// tcgen05 (5th-generation tensor core) helpers shared by the GEMM and the prefill attention:
// shared-memory matrix descriptors, the instruction descriptor of kind::f16, MMA issue and
// commit, tensor-memory loads.
#pragma once

#include "common.cuh"

namespace b200 {

// Tensor memory under programmatic launches. A kernel signals its dependents at its top and allocates its columns behind
// that, so a successor's CTA, with several kernels between them too, may allocate first and hold its columns while it
// waits for the very kernel that has yet to get its own. That cannot deadlock, because shared memory lets no more CTAs
// onto an SM (228 KB, 1 KB of it per CTA) than 512 columns serve: a kernel with tensor memory
//   takes so much that no other such kernel fits beside it (the smallest uses 45 KB),
//   or holds at most 256 columns and takes 105 KB, so that there are two of them, or one beside 122 KB of the rest,
//   or holds at most 128 columns per 105 KB: 276 on an SM, 148 in 122 KB.
constexpr bool tensor_memory_fits(int columns, int smem) {
  return smem >= 45 * 1024 && (smem > 182 * 1024 || (columns <= 256 && smem >= 105 * 1024) ||
                               columns * 105 <= 128 * (smem / 1024));
}

// Shared-memory matrix descriptor of a K-major tile of 128-byte swizzled rows: start address,
// leading byte offset 16 B (unused by swizzled K-major layouts), stride byte offset 1024 B
// (8 rows of 128 B per swizzle atom), descriptor version 1 (Blackwell), layout SWIZZLE_128B.
__device__ __forceinline__ uint64_t smem_descriptor(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4) | (uint64_t(1) << 16) |
         (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61);
}

// The same for an MN-major operand (rows of the tile are the K index, the 64 elements of a
// 128-byte swizzled row run along M or N): stride byte offset 1024 B between groups of 8 K
// rows, leading byte offset = distance between the 64-wide panels along M / N. One K step of
// 16 advances the start address by 16 rows = 2048 B. (Checked against a reference product.)
__device__ __forceinline__ uint64_t smem_descriptor_mn_major(uint32_t smem_addr,
                                                             uint32_t panel_stride_bytes) {
  return static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4) |
         (static_cast<uint64_t>(panel_stride_bytes >> 4) << 16) | (uint64_t(1024 >> 4) << 32) |
         (uint64_t(1) << 46) | (uint64_t(2) << 61);
}

// Instruction descriptor of kind::f16: fp32 accumulator, A and B both bf16 or (format 0) both fp16; each
// K-major, or MN-major (the transpose bits 15 of A and 16 of B).
__host__ __device__ constexpr uint32_t instruction_descriptor(int m, int n, bool b_mn_major = false,
                                                              bool a_mn_major = false, bool fp16 = false) {
  return (1u << 4) | (fp16 ? 0u : (1u << 7) | (1u << 10)) | (a_mn_major ? (1u << 15) : 0u) | (b_mn_major ? (1u << 16) : 0u) |
         (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// One product of 16 along K (M and N from the instruction descriptor). The issuing warp walks its loops as a whole, so
// that descriptors stay in uniform registers, and the one lane that passes a leader other than 0 issues (elect_one;
// always the same lane: a commit covers its own thread's products). A product of M 128 x N takes N / 2 cycles where
// N is wide and never less than some 40 (48 at N 64, 39 at N 16), dependent on the one before or not. A lone thread in a branch of its own could not issue
// that fast: 46 cycles a product, 57 with a commit behind every fourth, and its polls waited behind them. Projections on
// 128 rows x 64 columns a CTA, K 4864, 515 rows: 27.8 -> 24.4 us, 16 rows x 3584 x 3584 22.1 -> 17.3; 16384 rows, 128 x
// 256 columns a CTA, 234 -> 216 (9728 x 896).
__device__ __forceinline__ void umma_bf16_if(uint32_t leader, uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(leader)
      : "memory");
}
// The same with A in tensor memory: row r of A in lane r, K step of 16 in 8 columns of two neighbouring elements each.
__device__ __forceinline__ void umma_bf16_tmem_if(uint32_t leader, uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc,
                                                  uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(leader)
      : "memory");
}
__device__ __forceinline__ void umma_commit_if(uint32_t leader, uint32_t bar) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
               "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
               ::"r"(bar), "r"(leader) : "memory");
}

// 1 on one lane of a whole warp, 0 on the others: the lane that issues.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t leader;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(leader));
  return leader;
}
// A bounded wait of a whole warp, whose outcome is the same on all lanes.
__device__ __forceinline__ bool mbarrier_wait_warp(uint32_t bar, uint32_t parity, uint32_t limit) {
  return __all_sync(0xffffffffu, mbarrier_wait_ready_first(bar, parity, limit));
}
__device__ __forceinline__ bool mbarrier_spin_warp(uint32_t bar, uint32_t parity, uint32_t limit) {
  return __all_sync(0xffffffffu, mbarrier_spin_bounded(bar, parity, limit));
}

// The copies of a ring, from a warp that walks its loop as a whole as well: the announcement of a stage's bytes and the
// boxes, issued by the leader. From a lone thread, whose polls take 200 cycles more, a stage of 128 + 64 rows took longer
// to ask for than to multiply: 515 rows x 4864 x 896 24.4 -> 23.6 us, 32 rows of a Bazirax step 5190 -> 5101 us.
__device__ __forceinline__ void mbarrier_arrive_expect_tx_if(uint32_t leader, uint32_t bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
               "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %0;\n\t}" ::"r"(bytes), "r"(bar), "r"(leader)
               : "memory");
}
__device__ __forceinline__ void tma_load_2d_if(uint32_t leader, uint32_t dst, const void* tensor_map, uint32_t bar,
                                               int c0, int c1) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tensor_map)), "r"(bar), "r"(c0), "r"(c1), "r"(leader)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_if(uint32_t leader, uint32_t dst, const void* tensor_map, uint32_t bar,
                                               int c0, int c1, int c2) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];\n\t}"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tensor_map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(leader)
      : "memory");
}

__device__ __forceinline__ void tmem_load_32x32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_load_32x32(uint32_t taddr, float (&v)[16]) {  // 16 columns
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// The same load without its wait: several may be in flight. tmem_load_wait makes the values of
// one of them usable (the registers are operands of the wait, so nothing that reads them can be
// scheduled ahead of it).
__device__ __forceinline__ void tmem_load_32x32_issue(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_load_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                 "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]),
                 "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]),
                 "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                 "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]),
                 "+r"(r[31])
               :
               : "memory");
}

// 32 lanes x 32 columns back to tensor memory (each thread its own lane); tmem_store_wait
// before anything else may read them.
__device__ __forceinline__ void tmem_store_32x32(uint32_t taddr, const float (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
      ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]),
        "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]),
        "f"(v[15]), "f"(v[16]), "f"(v[17]), "f"(v[18]), "f"(v[19]), "f"(v[20]), "f"(v[21]),
        "f"(v[22]), "f"(v[23]), "f"(v[24]), "f"(v[25]), "f"(v[26]), "f"(v[27]), "f"(v[28]),
        "f"(v[29]), "f"(v[30]), "f"(v[31])
      : "memory");
}
// 16 columns of raw words
__device__ __forceinline__ void tmem_store_32x16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_store_32x32(uint32_t taddr, const float (&v)[16]) {  // 16 columns
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
      ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]),
        "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_store_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}

// A descriptor moved by a byte offset inside its tile (only the 14-bit start-address field
// changes as long as the tile stays below 256 KB).
__device__ __forceinline__ uint64_t descriptor_advance(uint64_t descriptor, uint32_t bytes) {
  return descriptor + (bytes >> 4);
}

}  // namespace b200
