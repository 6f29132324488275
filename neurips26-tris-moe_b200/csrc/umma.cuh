// tcgen05 (5th-generation tensor core) and TMEM primitives shared by the tensor-core kernels:
// shared-memory and instruction descriptors, MMA issue and commit, TMEM allocation and loads,
// and the cp.async staging of a row-major fp16 tile into the K-major no-swizzle core-matrix
// layout (8 rows x 16 bytes per core matrix; byte offset(row, k) =
// (k/8) * ROWS * 16 + row * 16 + (k%8) * 2; SBO = 128 B between 8-row groups, LBO = ROWS * 16 B
// between 8-column K chunks).
#pragma once
#include <cuda.h>  // CUtensorMap and its enums; cuTensorMapEncodeTiled itself comes from the driver entry point

#include "common.cuh"

namespace tris {

constexpr int kTcThreads = 128;
constexpr int kTcM = 128;   // outputs per tile = TMEM lanes
constexpr int kTcKChunk = 64;

__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  // start address [0,14) (>>4), leading byte offset [16,30) (>>4), stride byte offset [32,46) (>>4),
  // descriptor version 1 at [46,48), layout type 0 (no swizzle) at [61,64)
  return static_cast<uint64_t>((smem_addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16) |
         (static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// K-major, 128-byte swizzle: 1024 bytes between 8-row groups; a K = 16 step is 32 bytes further.
__device__ __forceinline__ uint64_t umma_smem_desc_sw128(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr >> 4) & 0x3FFFu) | (1ull << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) |
         (2ull << 61);
}

// kind::f16 instruction descriptor: fp16 A and B, both K-major, fp32 accumulate, M x N.
__device__ __forceinline__ uint32_t umma_idesc_f16(int m, int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ void umma_f16_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 lanes x 16 consecutive 32-bit columns of the accumulator: thread t of the warp gets lane
// (taddr.lane + t), registers = columns.
// The wait is part of the statement: nothing may touch the registers before it, not even a spill.
__device__ __forceinline__ void tmem_ld_16(uint32_t taddr, float (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
               : "r"(taddr)
               : "memory");
}
// Two of them with one wait.
__device__ __forceinline__ void tmem_ld_16_pair(uint32_t taddr_v, uint32_t taddr_w, float (&v)[16], float (&w)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n\t"
               "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n\ttcgen05.wait::ld.sync.aligned;"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]), "=f"(w[4]), "=f"(w[5]), "=f"(w[6]), "=f"(w[7]), "=f"(w[8]), "=f"(w[9]), "=f"(w[10]), "=f"(w[11]), "=f"(w[12]), "=f"(w[13]), "=f"(w[14]), "=f"(w[15])
               : "r"(taddr_v), "r"(taddr_w)
               : "memory");
}

// Twice 8 columns with one wait.
__device__ __forceinline__ void tmem_ld_8_pair(uint32_t taddr_v, uint32_t taddr_w, float (&v)[8], float (&w)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n\t"
               "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n\ttcgen05.wait::ld.sync.aligned;"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]), "=f"(w[4]), "=f"(w[5]), "=f"(w[6]), "=f"(w[7])
               : "r"(taddr_v), "r"(taddr_w)
               : "memory");
}

// Registers -> TMEM: thread t of the warp writes COUNT consecutive 32-bit columns of lane (taddr.lane + t).
// This is how a computed A operand gets to the tensor core without passing through shared memory: column
// c of lane m holds A[m][2c], A[m][2c + 1].
template <int COUNT>
__device__ __forceinline__ void tmem_st(uint32_t taddr, const uint32_t (&r)[COUNT]) {
  static_assert(COUNT == 8 || COUNT == 16, "columns per store");
  if constexpr (COUNT == 16)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
  else
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// A from TMEM (128 lanes, 8 columns per K = 16 step), B from shared memory.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Starts the asynchronous copy of a ROWS x 64 fp16 tile (row-major source, 128 B per row) into
// the core-matrix layout.  row_ptr(r) returns the source row (already offset to the chunk's
// first column) or nullptr for a row that must read as zeros.
// Only the first `valid_chunks` 8-column groups of the 64 columns exist in the source; the
// rest read as zeros.
template <int ROWS, typename RowPtr>
__device__ __forceinline__ void stage_operand_async(uint8_t* dst, const __half* fallback, RowPtr row_ptr,
                                                    int valid_chunks = 8) {
  constexpr int kVecs = ROWS * 8;
  for (int idx = threadIdx.x; idx < kVecs; idx += blockDim.x) {
    // a warp covers 8 rows x 4 chunks: 64 contiguous source bytes per row, and every 8
    // consecutive lanes write 128 contiguous shared-memory bytes
    const int r_lo = idx & 7, c_lo = (idx >> 3) & 3, rest = idx >> 5;
    const int c = ((rest & 1) << 2) | c_lo, row = ((rest >> 1) << 3) | r_lo;
    const __half* src = row_ptr(row);
    const bool valid = src != nullptr && c < valid_chunks;
    cp_async_16(dst + (c * ROWS + row) * 16, valid ? src + 8 * c : fallback, valid);
  }
}

__device__ __forceinline__ void tma_load_2d(void* dst_smem, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                   smem_u32(dst_smem)),
               "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
               : "memory");
}
// Describes row-major fp16 rows of `cols` columns, `stride` halves apart (multiples of 8, `base` at a 16-byte boundary);
// one copy = one 64-column chunk of box_rows rows, 128-byte-swizzled, zeros past the matrix (tc_gemm.cu).
bool encode_rows_map(CUtensorMap* map, const void* base, int rows, int cols, int stride, int box_rows);

}  // namespace tris
