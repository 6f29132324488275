// Tile records: the load-time, tile-major image of a block-GR compact3 projection, and the device
// code that turns it into fp16 tensor-core operands.  Shared by the record builder, the grouped
// kernels and the dequantising dump kernel, so that the bit-exact parity checks run the code of the
// hot path.
//
// Why records.  The E-stacked payload tensors of build_grouped_precomputed_payload (QL:1512-1636 of
// the TriS-MoE tree) are laid out plane by plane and the grouping bits are Golomb-Rice coded.  A
// kernel that reads them pays, per weight, for the decode (4 lane-instructions of a serial
// codeword chain) and for a bit layout that does not match the fragment it wants.  A record holds
// the same information decoded once, at load time, as 2 bits per weight in the order the unpack
// consumes them.  That is 1 bit of grouping plane against 0.47 bits of code plus 0.25 bits of
// sub-stream index (what a parallel decode needs): 12 % more record bytes for a quarter of the
// instructions.
//
//   tile record (expert e, outputs 128*tile .. +127, columns 128*chunk .. +127): four sub-records of 32
//   outputs each, so that any run of 32-output groups is one contiguous piece; a sub-record is
//     codes    512 B per 64-column slice: [slice][output] 16 B = 4 code words of 16 columns
//     sal      128 B per salient step:    [step][output] 4 B = 16 salient columns, two sign bits each
//     rows     256 B per row-scale slot:  [slot][output] 8 B = row_pack3 word (s_r1, s_r2, ns_d, ns_nd)
//   All records of a projection have the same size (TrisProjView.max_record_bytes), so a record is
//   found without a table.
//
//   column record (expert e, chunk), shared by all output tiles
//     header    64 B  slot of every packed row, slot of every salient step
//     coltab   512 B  per column pair the (ns_d, ns_nd) scales as two half2, zero at salient columns;
//                     [slice][pairs 2j, 2j + 1 of a code word][code word] 16 B
//     steps     96 B  per salient step: 8 pairs of (s_c1, s_c2) half2, then the 16 columns (uint16)
//
// Code word of columns 16w .. 16w+15: w << i (i = 0..7) holds, for columns 2i / 2i+1, the negative-sign
// bits at 15 / 31 and the grouping bits at 7 / 23.  One shift therefore yields the sign of a half2
// in place and, through PRMT's sign-replicate mode, its select mask.  The code word of a salient step
// has the second sign at 7 / 23.
//
// A "row-scale slot" is a run of packed rows of the chunk that share one quantisation group (g_idx is
// constant inside a packed word; tris_build_row_groups checks that); with the usual groups of 128
// columns a chunk has one.  Salient columns (10 %) carry two signed terms.  The main unpack leaves +-0
// there, and a "salient step" - 16 salient columns of one slot, compacted - is multiplied as K columns
// of its own (one K = 16 MMA step) with gathered activations: fewer instructions per weight than
// patching them in place (0.6 against 2.3).
#pragma once
#include "common.cuh"

namespace tris {
namespace tr {

constexpr int kTileOut = 128;       // outputs per tile record = threads per unpacking warpgroup = TMEM lanes
constexpr int kChunkRows = 4;       // packed rows per record
constexpr int kChunkCols = 32 * kChunkRows;
constexpr int kSliceCols = 64;      // columns per 16-byte code group
constexpr int kSubOut = 32, kSubs = kTileOut / kSubOut;  // sub-records of a tile
constexpr int kSliceBytes = kSubOut * 16;                // within a sub-record
constexpr int kStepBytes = kSubOut * 4;
constexpr int kSlotBytes = kSubOut * 8;
constexpr int kMaxSteps = kChunkCols / 16;  // all columns salient
constexpr int kColHdrBytes = 64;
constexpr int kColTabBytes = kChunkCols * 4;
constexpr int kColStepBytes = 96;
constexpr uint32_t kColMagic = 0x33305254u;  // "TR03": layout version, checked when stored records are adopted

struct ColHeader {                  // 64 bytes; the unpack reads the first 20 as words
  uint32_t magic;
  uint8_t num_slots, num_steps;
  uint16_t num_salient;
  uint8_t slot_of_row[kChunkRows];
  uint8_t step_slot[kMaxSteps];
  uint32_t pad[11];
};
static_assert(kChunkRows == 4 && kMaxSteps == 8, "header words: counts at 1, packed rows at 2, steps at 3 and 4");
static_assert(sizeof(ColHeader) == kColHdrBytes, "column record header");

__host__ __device__ inline int tiles_per_expert(int out_features) { return (out_features + kTileOut - 1) / kTileOut; }
__host__ __device__ inline int num_chunks(int rank) { return ((rank + 31) / 32 + kChunkRows - 1) / kChunkRows; }
__host__ __device__ inline int col_record_bytes(int max_steps) { return kColHdrBytes + kColTabBytes + max_steps * kColStepBytes; }
// 64-column slices of a record: those the projection has, at most a chunk's two
__host__ __device__ inline int record_slices(int rank) {
  const int s = (rank + kSliceCols - 1) / kSliceCols;
  return s < kChunkCols / kSliceCols ? s : kChunkCols / kSliceCols;
}
__host__ __device__ inline int record_bytes(int rank, int max_steps, int max_slots) {
  return kSubs * (record_slices(rank) * kSliceBytes + max_steps * kStepBytes + max_slots * kSlotBytes);
}

// ---- salient step assignment ------------------------------------------------------------------
// One thread walks the chunk's packed rows.  A run of equal group ids is a row-scale slot.  Salient columns of a run
// fill steps of 16; a new run starts a new step.
struct ChunkPlan {
  int num_slots, num_steps;
};
__device__ inline ChunkPlan plan_chunk(const int32_t* c_map_e, const int32_t* row_group_e, int pr, int p0, int rank) {
  ChunkPlan plan{0, 0};
  int prev_group = -0x7fffffff, fill = 0;  // fill: salient columns of the run so far
  for (int p = p0; p < min(pr, p0 + kChunkRows); ++p) {
    const int grp = row_group_e ? row_group_e[p] : 0, ncols = rank - 32 * p;
    if (grp != prev_group) {
      prev_group = grp;
      ++plan.num_slots;
      fill = 0;
    }
    const int n = __popc(static_cast<uint32_t>(c_map_e[p]) & (ncols >= 32 ? ~0u : (ncols <= 0 ? 0u : (1u << ncols) - 1u)));
    plan.num_steps += (fill + n + 15) / 16 - (fill + 15) / 16;
    fill += n;
  }
  if (plan.num_slots == 0) plan.num_slots = 1;
  return plan;
}

// ---- register unpack ----------------------------------------------------------------------------
// Thread = output row.  The column scales are the same for all threads (broadcast shared-memory
// loads), the row scales are the thread's own.  Per half2 of two columns: a shift, a PRMT mask, two
// HMUL2, a select and a sign flip: 3.2 lane-instructions per weight with the scale loads.  Exact
// arithmetic of _dequantize_compact3_matrix (QL:4200-4236): one product per weight, rounded to
// fp16 once.
struct RowScales {
  __half2 rd, rn;  // ns_d_r1, ns_nd_r1 in both halves
};
__device__ __forceinline__ RowScales row_scales_ns(uint2 rp) {
  RowScales r;
  r.rd = u32_as_h2(prmt(rp.y, 0u, 0x1010u));
  r.rn = u32_as_h2(prmt(rp.y, 0u, 0x3232u));
  return r;
}

__device__ __forceinline__ uint32_t lop3_select(uint32_t a, uint32_t b, uint32_t m) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xCA;" : "=r"(d) : "r"(m), "r"(a), "r"(b));  // m ? a : b
  return d;
}
__device__ __forceinline__ uint32_t flip_by_sign(uint32_t v, uint32_t t) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0x78;" : "=r"(d) : "r"(v), "r"(t), "r"(0x80008000u));  // v ^ (t & mask)
  return d;
}

// Two half2 (columns 2i .. 2i + 3 of a code word w) of one output; t0 = w << i, t1 = w << (i + 1), c = {d, nd} scale words of
// the two pairs.
__device__ __forceinline__ void unpack_two(uint32_t t0, uint32_t t1, const uint4& c, const RowScales& rs, uint32_t& a, uint32_t& b) {
  const uint32_t d0 = h2_as_u32(__hmul2_rn(u32_as_h2(c.x), rs.rd)), n0 = h2_as_u32(__hmul2_rn(u32_as_h2(c.y), rs.rn));
  const uint32_t d1 = h2_as_u32(__hmul2_rn(u32_as_h2(c.z), rs.rd)), n1 = h2_as_u32(__hmul2_rn(u32_as_h2(c.w), rs.rn));
  a = flip_by_sign(lop3_select(d0, n0, prmt(t0, 0u, 0xAA88u)), t0);
  b = flip_by_sign(lop3_select(d1, n1, prmt(t1, 0u, 0xAA88u)), t1);
}

// 16 columns (code word i of a slice) -> 8 half2 in column order.  ct: the slice's scale table + i.
__device__ __forceinline__ void unpack_word(uint32_t w, const uint4* ct, const RowScales& rs, uint32_t* a) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint4 c = ct[4 * j];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t t = w << (2 * j + h);
      const uint32_t vd = h2_as_u32(__hmul2_rn(u32_as_h2(h ? c.z : c.x), rs.rd));
      const uint32_t vn = h2_as_u32(__hmul2_rn(u32_as_h2(h ? c.w : c.y), rs.rn));
      // grouping bit 1 -> "d" pair (CU:736-737); a clear sign-plane bit is a minus (QL:4213)
      a[2 * j + h] = flip_by_sign(lop3_select(vd, vn, prmt(t, 0u, 0xAA88u)), t);
    }
  }
}

// One salient step (16 columns) -> 8 half2: fp16(+-fp16(c1 r1) +- fp16(c2 r2)).
__device__ __forceinline__ void unpack_step(uint32_t w, const uint4* sc, uint2 rp, uint32_t* a) {
  const __half2 r1 = u32_as_h2(prmt(rp.x, 0u, 0x1010u)), r2 = u32_as_h2(prmt(rp.x, 0u, 0x3232u));
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint4 c = sc[j];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t t = w << (2 * j + h);
      const uint32_t p1 = flip_by_sign(h2_as_u32(__hmul2_rn(u32_as_h2(h ? c.z : c.x), r1)), t);
      const uint32_t p2 = flip_by_sign(h2_as_u32(__hmul2_rn(u32_as_h2(h ? c.w : c.y), r2)), t << 8);
      a[2 * j + h] = h2_as_u32(__hadd2_rn(u32_as_h2(p1), u32_as_h2(p2)));
    }
  }
}

// ---- finding records ------------------------------------------------------------------------------
struct RecordGeom {  // offsets inside a sub-record; rec_bytes and sub_bytes are sizes
  int32_t rec_bytes, sub_bytes, slices, chunks, tiles, sal_off, rows_off, slots, col_bytes;
};
__host__ __device__ inline RecordGeom record_geom(const TrisProjView& v) {
  RecordGeom g;
  g.rec_bytes = v.max_record_bytes;
  g.sub_bytes = v.max_record_bytes / kSubs;
  g.slices = record_slices(v.rank);
  g.chunks = num_chunks(v.rank);
  g.tiles = tiles_per_expert(v.out_features);
  g.sal_off = g.slices * kSliceBytes;
  g.rows_off = g.sal_off + v.max_sal_words * kStepBytes;
  g.slots = (g.sub_bytes - g.rows_off) / kSlotBytes;
  g.col_bytes = v.col_record_bytes;
  return g;
}
__device__ __forceinline__ const uint8_t* tile_record(const TrisProjView& v, const RecordGeom& g, int expert, int tile, int chunk) {
  return static_cast<const uint8_t*>(v.tile_records) +
         (static_cast<size_t>(expert * g.tiles + tile) * g.chunks + chunk) * static_cast<size_t>(g.rec_bytes);
}
__device__ __forceinline__ const uint8_t* col_record(const TrisProjView& v, const RecordGeom& g, int expert, int chunk) {
  return static_cast<const uint8_t*>(v.col_records) + static_cast<size_t>(expert * g.chunks + chunk) * static_cast<size_t>(g.col_bytes);
}
__device__ __forceinline__ uint4 ldg_stream(const void* p) {  // read once: do not keep it in L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

}  // namespace tr
}  // namespace tris
