// Grouped compact3 dequant-matmul over tile records for segments of few rows (decode), on mma.sync; also for a few
// segments of up to 128 rows, whose passes CTAs share.
//
// A warp owns 32 outputs of one projection and multiplies them with up to 8 NT activation rows.  Lane
// (g, t) takes code word t of output rows g, g + 8, g + 16, g + 24: 16 columns of each of a 64-column slice.
// Unpacked, they are the lane's A fragments of four m16n8k16 steps if step j's K positions are columns
// 16t + 4j .. + 3, which the B side follows: a lane's activations of a slice are 32 contiguous bytes.
// Weights go from the code words to the MMA in registers.
// tcgen05 tiles have 128 outputs and take their A from TMEM: allocation, stores and the hand-over to
// the issuing thread cost more than the unpack at a few rows per weight.
//
// Everything a CTA reads - code words, scales, tables, activation rows - is asked for at its start by
// cp.async and read from shared memory, so that the inner loop waits for nothing further away: with the
// same loop on L1 / L2 loads half the stall cycles were theirs.  (Bulk copies issued by the
// lanes of a warp take turns: gate/up and down of 64 experts, both forms timed in one run, 5.8 / 4.8 us at 1 token against
// 5.6 / 4.5, 14.0 / 13.4 at 32 against 14.0 / 12.7, but 21.4 / 20.5 at 128 against 23.4 / 20.1.)
// What bounds it now (128 tokens of 64 experts, 20.9 / 18.6 us): latency at four warps per scheduler.  An instruction issues
// in 55 / 57 % of the cycles; a warp waits 21 % of its time for fixed latencies, 17 % for the loads at a unit's start, 11 %
// for the tensor pipe.  1024 CTAs over 740 slots are 1.4 waves.
//
// CTAs are small (four warps, five to seven CTAs per SM), so that the units of a decode batch are nearly
// all resident at once and SMs are evenly loaded.  With few units the columns are split over KS warps
// (partial sums added through shared memory): whole 128-column chunks over KS = 2, 64-column halves over KS = 4.
// Matrices of many columns and few outputs: the CTAs of a cluster take column parts of the same outputs too, and each
// finishes its share of the sums from the others' shared memory (no scratch, no atomics, always the same order).
#include <cooperative_groups.h>

#include "grouped_tiled.cuh"

namespace cg = cooperative_groups;

namespace tris {
namespace tr {

constexpr int kDecOut = 32;                                                  // outputs of a warp
constexpr int dec_warps(int proj, int ks) { return proj * ks > 4 ? proj * ks : 4; }
constexpr int dec_groups(int proj, int ks) { return dec_warps(proj, ks) / (proj * ks); }
constexpr int kDecCols = 256;                     // columns staged at a time
constexpr int kDecRowBytes = 2 * kDecCols + 16;  // odd multiple of 16: conflict-free
// One buffer: [projection][chunk]{sub-records of the CTA's outputs, column record}, then [set][8 NT rows]
struct DecodeLayout {
  int col_off, chunk_bytes, acts_off, acts_bytes, total;
};
__host__ __device__ inline DecodeLayout decode_layout(int max_sub_bytes, int max_steps, int nproj, int nset, int nt, int ks) {
  DecodeLayout l;
  l.col_off = dec_groups(nproj, ks) * max_sub_bytes;
  l.chunk_bytes = l.col_off + col_record_bytes(max_steps);
  l.acts_off = nproj * (kDecCols / kChunkCols) * l.chunk_bytes;
  l.acts_bytes = 8 * nt * kDecRowBytes;
  l.total = l.acts_off + nset * l.acts_bytes;
  return l;
}

// Warps that an SM should hold; a launch with column parts has no more than 14 for it.
constexpr int dec_min_ctas(int nt, int warps, bool parts) { return (parts ? 16 : (nt <= 2 ? 28 : 20)) / warps; }

// grid (groups of 32 * dec_groups outputs, segments, CTAs that share a segment's passes or, as a cluster, its columns)
template <int NT, int MODE, int KS, bool kParts>
__global__ void __launch_bounds__(32 * dec_warps(MODE == MODE_SINGLE ? 1 : 2, KS), dec_min_ctas(NT, dec_warps(MODE == MODE_SINGLE ? 1 : 2, KS), kParts))
    grouped_decode_kernel(const __grid_constant__ TiledArgs args) {
  constexpr bool DUAL = MODE != MODE_SINGLE;
  constexpr int P = DUAL ? 2 : 1;
  constexpr int NW = dec_warps(P, KS), OG = dec_groups(P, KS), kThreads = 32 * NW;
  constexpr bool HALF = KS >= 4;                         // a warp takes one half of a chunk
  constexpr int CS = HALF ? KS / 2 : KS;                 // chunks are dealt to CS warps
  constexpr int kCols = kDecCols, kRow = kDecRowBytes;
  constexpr int kGroupChunks = kCols / kChunkCols;
  extern __shared__ uint4 smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>(smem_raw);

  if (!args.weights_before_wait) {
    pdl_wait();
    pdl_launch_dependents();
  }
  const int seg = blockIdx.y;
  const int nseg = args.num_segments_dev ? min(*args.num_segments_dev, args.num_segments) : args.num_segments;
  // A CTA without rows leaves at once, but the first one waits: if none did, the launch could end before its predecessor.
  auto leave = [&]() {
    if (args.weights_before_wait && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) pdl_wait();
  };
  if (seg >= nseg) return leave();
  const int expert = args.expert_ids ? args.expert_ids[seg] : 0;  // no arrays: one segment of expert 0 with all rows
  // kParts: args.col_split neighbours along z, a cluster, share the columns
  const int part = kParts ? static_cast<int>(blockIdx.z) % args.col_split : 0, first_pass = kParts ? static_cast<int>(blockIdx.z) / args.col_split : blockIdx.z;
  const int row_begin = (args.expert_ids ? args.segment_offsets[seg] : 0) + first_pass * 8 * NT;
  const int row_end = args.expert_ids ? min(args.segment_offsets[seg + 1], args.num_rows) : args.num_rows;
  if (expert < 0 || expert >= args.num_experts || row_end <= row_begin) return leave();

  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int p = DUAL ? warp & 1 : 0, og = (warp / P) % OG, ks = warp / (P * OG);
  const int hs = HALF ? (ks & 1) : 0, first_chunk = HALF ? (ks >> 1) : ks;
  const int cta_o = blockIdx.x * OG * kDecOut, o0 = cta_o + og * kDecOut;
  const bool mine = o0 < args.out_features;
  const TrisProjView& v = args.proj[p];
  const int sub_bytes = v.max_record_bytes / kSubs, sal_off = record_slices(args.rank) * kSliceBytes, rows_off = sal_off + v.max_sal_words * kStepBytes;
  const DecodeLayout L = decode_layout(args.max_sub_bytes, args.max_steps, P, args.num_sets, NT, KS);
  int gr_begin = 0, gr_end = (args.rank + kCols - 1) / kCols;
  if (kParts) {
    const int all = gr_end;
    gr_begin = part * all / args.col_split;
    gr_end = (part + 1) * all / args.col_split;
  }
  const bool ring = args.stages > 1;  // two buffers
  auto buffer = [&](int b) { return sm + b * L.total; };

  // Records of column group gr: per projection and chunk one linear run each of the tile and column record.
  auto stage_weights = [&](int gr, int b) {
    const int chunks = min(kGroupChunks, args.chunks - gr * kGroupChunks);
    const int tile = cta_o / kTileOut, sub = (cta_o % kTileOut) / kSubOut;
#pragma unroll 1
    for (int pp = 0; pp < P; ++pp) {
      const TrisProjView& pv = args.proj[pp];
      const int rec_bytes = pv.max_record_bytes, run = OG * (rec_bytes / kSubs), col_bytes = pv.col_record_bytes;
      const int c = gr * kGroupChunks;
      const uint8_t* rec = static_cast<const uint8_t*>(pv.tile_records) + sub * (rec_bytes / kSubs) +
                           static_cast<size_t>((expert * args.tiles + tile) * args.chunks + c) * static_cast<size_t>(rec_bytes);
      const uint8_t* col = static_cast<const uint8_t*>(pv.col_records) + static_cast<size_t>(expert * args.chunks + c) * static_cast<size_t>(col_bytes);
      uint8_t* dst = buffer(b) + pp * kGroupChunks * L.chunk_bytes;
#pragma unroll 1
      for (int ch = 0; ch < chunks; ++ch, rec += rec_bytes, col += col_bytes, dst += L.chunk_bytes) {
        for (int i = tid * 16; i < run; i += kThreads * 16) cp_async_16(dst + i, rec + i);
        for (int i = tid * 16; i < col_bytes; i += kThreads * 16) cp_async_16(dst + L.col_off + i, col + i);
      }
    }
  };
  // Activation rows r0 .. of column group gr, zero up to a multiple of 64 columns.
  auto stage_acts = [&](int gr, int b, int r0, int rows) {
    const int c0 = gr * kCols, cols = min(kCols, args.rank - c0);
    const int pieces = ((cols + kSliceCols - 1) / kSliceCols) * (kSliceCols / 8);
    constexpr int kPieces = kCols / 8, kStep = kThreads / kPieces;
    const int piece = tid % kPieces, left = cols - 8 * piece;
    if (piece < pieces) {
      uint8_t* d = buffer(b) + L.acts_off + (tid / kPieces) * kRow + piece * 16;
      const int at = c0 + (left > 0 ? 8 * piece : 0);
#pragma unroll 2
      for (int n = tid / kPieces; n < rows; n += kStep, d += kStep * kRow) {
        const int src = args.row_gather ? args.row_gather[r0 + n] : r0 + n;
        const size_t off = static_cast<size_t>(src) * args.hidden_stride;
        if (args.hidden_vec) {
          cp_async_16(d, args.hidden[0] + off + at, left > 0);
          if (P == 2 && args.num_sets == 2) cp_async_16(d + L.acts_bytes, args.hidden[1] + off + at, left > 0);
        } else {
          *reinterpret_cast<uint4*>(d) = read_piece(args, args.hidden[0] + off + c0, c0, piece, left);
          if (P == 2 && args.num_sets == 2) *reinterpret_cast<uint4*>(d + L.acts_bytes) = read_piece(args, args.hidden[1] + off + c0, c0, piece, left);
        }
      }
    }
    cp_async_commit();
  };

  stage_weights(gr_begin, 0);
  if (args.weights_before_wait) {
    if (!kParts || !args.rows_ready) pdl_wait();
    pdl_launch_dependents();
  }

  // Whether this CTA of a cluster writes rows 8 nt .. of outputs 16 m ..
  auto finishes = [&](int m, int nt) { return !kParts || (2 * nt + m) % args.col_split == part; };
  int load = 0;  // column groups loaded so far
#pragma unroll 1
  for (int r0 = row_begin; r0 < row_end; r0 += 8 * NT * args.row_split) {
    const int rows = min(8 * NT, row_end - r0);
    float acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[m][nt][c] = 0.f;
    {
      const int b = ring ? load & 1 : 0;
      if (r0 != row_begin) {  // the previous pass has read its buffers and partial sums
        if constexpr (kParts) cg::this_cluster().sync();
        else __syncthreads();
        stage_weights(gr_begin, b);
      }
      stage_acts(gr_begin, b, r0, rows);
    }
#pragma unroll 1
    for (int gr = gr_begin; gr < gr_end; ++gr, ++load) {
      const int b = ring ? load & 1 : 0;
      cp_async_wait<0>();
      __syncthreads();
      if (gr + 1 < gr_end) {  // the other buffer was read before the barrier
        stage_weights(gr + 1, b ^ 1);
        stage_acts(gr + 1, b ^ 1, r0, rows);
      }
      if (!mine) continue;
      const uint8_t* rows_buf = buffer(b) + L.acts_off + (args.num_sets == 2 ? p : 0) * L.acts_bytes + g * kRow;
      const int chunks = min(kGroupChunks, args.chunks - gr * kGroupChunks);
#pragma unroll 1
      for (int ch = first_chunk; ch < chunks; ch += CS) {
        const uint8_t* ck = buffer(b) + (p * kGroupChunks + ch) * L.chunk_bytes;
        const uint8_t* col = ck + L.col_off;
        const uint8_t* sub = ck + og * sub_bytes;
        const uint8_t* scales = sub + rows_off + g * 8;
        const uint8_t* x_base = rows_buf + ch * (kChunkCols * 2);
        const int cols = args.rank - (gr * kGroupChunks + ch) * kChunkCols;     // from here on
        const uint32_t counts = reinterpret_cast<const uint32_t*>(col)[1];       // ColHeader: slots, steps << 8
        const bool several = (counts & 0xFFu) > 1u;  // row-scale slots in the chunk (groups of fewer than 128 columns)
        RowScales rs[4];
        auto load_scales = [&](int slot) {
#pragma unroll
          for (int i = 0; i < 4; ++i) rs[i] = row_scales_ns(*reinterpret_cast<const uint2*>(scales + slot * kSlotBytes + i * 64));
        };
        load_scales(0);
#pragma unroll 1
        for (int sl = hs; sl < (HALF ? hs + 1 : 2) && sl * kSliceCols < cols; ++sl) {
          if (several) load_scales(col[8 + 2 * sl + (t >> 1)]);  // ColHeader.slot_of_row of the lane's packed row
          const uint8_t* cw = sub + sl * kSliceBytes + g * 16 + t * 4;
          uint32_t cur[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) cur[i] = *reinterpret_cast<const uint32_t*>(cw + i * 128);
          const uint4* ct = reinterpret_cast<const uint4*>(col + kColHdrBytes) + sl * 16 + t;
          const uint8_t* x = x_base + sl * (kSliceCols * 2) + t * 32;
#pragma unroll
          for (int jj = 0; jj < 2; ++jj) {
            uint4 bf[NT];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) bf[nt] = *reinterpret_cast<const uint4*>(x + nt * 8 * kRow + jj * 16);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const uint4 cs = ct[(2 * jj + j) * 4];
#pragma unroll
              for (int m = 0; m < 2; ++m) {
                uint32_t a0, a1, a2, a3;
                unpack_two(cur[2 * m] << (4 * jj + 2 * j), cur[2 * m] << (4 * jj + 2 * j + 1), cs, rs[2 * m], a0, a2);
                unpack_two(cur[2 * m + 1] << (4 * jj + 2 * j), cur[2 * m + 1] << (4 * jj + 2 * j + 1), cs, rs[2 * m + 1], a1, a3);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
                  mma_m16n8k16(acc[m][nt], a0, a1, a2, a3, j ? bf[nt].z : bf[nt].x, j ? bf[nt].w : bf[nt].y);
              }
            }
          }
        }
        // salient steps: lane t takes pairs 2t, 2t + 1 of the step's 16 columns
        const int steps = static_cast<int>((counts >> 8) & 0xFFu);
#pragma unroll 1
        for (int st = hs; st < steps; st += HALF ? 2 : 1) {
          const uint8_t* ent = col + kColHdrBytes + kColTabBytes + st * kColStepBytes;
          const uint8_t* wsrc = sub + sal_off + st * kStepBytes + g * 4;
          const uint8_t* rsrc = scales + (several ? col[12 + st] : 0) * kSlotBytes;  // ColHeader.step_slot
          const uint4 cs = reinterpret_cast<const uint4*>(ent)[t];
          const uint2 at = reinterpret_cast<const uint2*>(ent + 64)[t];
          uint32_t bf[NT][2];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            auto ld = [&](uint32_t cc) -> uint32_t { return *reinterpret_cast<const uint16_t*>(x_base + 2 * cc + nt * 8 * kRow); };
            bf[nt][0] = prmt(ld(at.x & 0xFFFFu), ld(at.x >> 16), 0x5410u);
            bf[nt][1] = prmt(ld(at.y & 0xFFFFu), ld(at.y >> 16), 0x5410u);
          }
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            uint32_t a[2][2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint32_t w = *reinterpret_cast<const uint32_t*>(wsrc + (2 * m + h) * 32) << (2 * t);
              const uint32_t rp = *reinterpret_cast<const uint32_t*>(rsrc + (2 * m + h) * 64);
              const __half2 r1 = u32_as_h2(prmt(rp, 0u, 0x1010u)), r2 = u32_as_h2(prmt(rp, 0u, 0x3232u));
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const uint32_t tt = w << i;
                const uint32_t p1 = flip_by_sign(h2_as_u32(__hmul2_rn(u32_as_h2(i ? cs.z : cs.x), r1)), tt);
                const uint32_t p2 = flip_by_sign(h2_as_u32(__hmul2_rn(u32_as_h2(i ? cs.w : cs.y), r2)), tt << 8);
                a[h][i] = h2_as_u32(__hadd2_rn(u32_as_h2(p1), u32_as_h2(p2)));
              }
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_m16n8k16(acc[m][nt], a[0][0], a[1][0], a[0][1], a[1][1], bf[nt][0], bf[nt][1]);
          }
        }
      }
    }

    // Output scale and bias act on the whole sum: applied to the first part, the bias once.
    if (mine && (v.output_scale || v.bias)) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const size_t at = static_cast<size_t>(expert) * args.out_features + min(o0 + g + 8 * i, args.out_features - 1);
        const float scale = v.output_scale ? __half2float(static_cast<const __half*>(v.output_scale)[at]) : 1.f;
        const float bias = v.bias && ks == 0 && part == 0 ? __half2float(static_cast<const __half*>(v.bias)[at]) : 0.f;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) acc[i >> 1][nt][2 * (i & 1) + e] = acc[i >> 1][nt][2 * (i & 1) + e] * scale + bias;
      }
    }
    // Partial sums meet: 16 outputs m of a pair of warps are finished by the gate warp (m = 0) or the up warp
    // (m = 1) for SiLU(gate) * up, by each projection's own warp otherwise; always by the ks = 0 warp.
    float up[NT][4];
    if constexpr (KS > 1 || MODE == MODE_DUAL_SILU) {
      float4* sums = reinterpret_cast<float4*>(sm);
      auto slot_of = [&](int pp, int kk, int m, int nt) { return sums + (((((pp * KS + kk) * OG + og) * 2 + m) * NT + nt) * 32 + lane); };
      __syncthreads();  // every warp is done with the activation rows
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        if (ks == 0 && (MODE != MODE_DUAL_SILU || m == p || kParts)) continue;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) *slot_of(p, ks, m, nt) = make_float4(acc[m][nt][0], acc[m][nt][1], acc[m][nt][2], acc[m][nt][3]);
      }
      __syncthreads();
      if (ks > 0 && !kParts) continue;
      auto add = [&](float (&x)[4], const float4* q) {
        const float4 y = *q;
        x[0] += y.x;
        x[1] += y.y;
        x[2] += y.z;
        x[3] += y.w;
      };
      if constexpr (kParts) {
        // sums of this CTA's columns, then of the cluster's: a CTA finishes every col_split-th eight rows of 16 outputs
        cg::cluster_group cluster = cg::this_cluster();
        if (ks == 0) {
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
              for (int k = 1; k < KS; ++k) add(acc[m][nt], slot_of(p, k, m, nt));
              *slot_of(p, 0, m, nt) = make_float4(acc[m][nt][0], acc[m][nt][1], acc[m][nt][2], acc[m][nt][3]);
            }
        }
        cluster.sync();
        if (ks > 0 || !mine) continue;
        auto total = [&](float (&x)[4], int pp, int m, int nt) {
#pragma unroll
          for (int e = 0; e < 4; ++e) x[e] = 0.f;
#pragma unroll 4
          for (int z = 0; z < args.col_split; ++z) add(x, cluster.map_shared_rank(slot_of(pp, 0, m, nt), z));
        };
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          if constexpr (MODE == MODE_DUAL_SILU) {
            if (!finishes(p, nt)) continue;
            total(acc[0][nt], p, p, nt);
            total(up[nt], p ^ 1, p, nt);
          } else {
#pragma unroll
            for (int m = 0; m < 2; ++m)
              if (finishes(m, nt)) total(acc[m][nt], p, m, nt);
          }
        }
      } else {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          if constexpr (MODE == MODE_DUAL_SILU) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (p) acc[0][nt][e] = acc[1][nt][e];  // the finished half is m = p
              up[nt][e] = 0.f;
            }
#pragma unroll
            for (int k = 1; k < KS; ++k) add(acc[0][nt], slot_of(p, k, p, nt));
#pragma unroll
            for (int k = 0; k < KS; ++k) add(up[nt], slot_of(p ^ 1, k, p, nt));
          } else {
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
              for (int k = 1; k < KS; ++k) add(acc[m][nt], slot_of(p, k, m, nt));
          }
        }
      }
    }
    if (!mine) continue;

    if (kParts && args.rows_ready) pdl_wait();
    // epilogue: a 16-output half holds {(output g, row 2t), (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1)}
    constexpr int kHalves = MODE == MODE_DUAL_SILU ? 1 : 2;
#pragma unroll
    for (int m = 0; m < kHalves; ++m) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        if (nt * 8 < rows && finishes(MODE == MODE_DUAL_SILU ? p : m, nt)) {
          float y[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            y[e] = acc[m][nt][e];
            if constexpr (MODE == MODE_DUAL_SILU) {
              const float gate = p ? up[nt][e] : y[e], lin = p ? y[e] : up[nt][e];
              y[e] = __fdividef(gate, 1.f + __expf(-gate)) * lin;
            }
          }
          // transposed: this lane holds row g, outputs 2t, 2t + 1 (lo) and 8 + 2t, 9 + 2t (hi); neighbours swap one
          // so that each stores four outputs
          const uint2 w = outputs_of_row(h2_as_u32(__floats2half2_rn(y[0], y[1])), h2_as_u32(__floats2half2_rn(y[2], y[3])), t);
          const int n = nt * 8 + g;
          const int orow = n >= rows ? -1 : (args.out_scatter ? args.out_scatter[r0 + n] : r0 + n);
          if (orow >= 0) {
            const int o = o0 + 16 * (MODE == MODE_DUAL_SILU ? p : m) + ((t & 1) ? 8 : 0) + 2 * (t & 2);
            __half* dst = args.out[MODE == MODE_DUAL_STORE ? p : 0] + static_cast<size_t>(orow) * args.out_features + o;
            if (args.quad_store) {
              if (o < args.out_features) *reinterpret_cast<uint2*>(dst) = w;
            } else {
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (o + i < args.out_features)
                  dst[i] = __ushort_as_half(static_cast<unsigned short>((i & 2 ? w.y : w.x) >> (16 * (i & 1))));
            }
          }
          __syncwarp();  // the transposes need the warp together
        }
      }
    }
  }
  if constexpr (kParts) cg::this_cluster().sync();  // shared memory stays until the others have read their sums
}

template <int NT, int MODE, int KS, bool kParts = false>
static int launch_decode(TiledArgs args, cudaStream_t stream, bool pdl, int col_split = 1) {
  constexpr int P = MODE == MODE_SINGLE ? 1 : 2;
  args.col_split = col_split;
  args.stages = args.rank > kDecCols * col_split ? 2 : 1;  // col_split is no more than there are groups: every CTA has one
  const int part = (KS > 1 || MODE == MODE_DUAL_SILU) ? dec_warps(P, KS) * 2 * NT * 512 : 0;
  const size_t smem = std::max(args.stages * decode_layout(args.max_sub_bytes, args.max_steps, P, args.num_sets, NT, KS).total, part);
  TRIS_REQUIRE(smem <= kMostSmem, TRIS_ERR_UNSUPPORTED, "grouped_decode_kernel: %zu bytes of shared memory", smem);
  auto kernel = grouped_decode_kernel<NT, MODE, KS, kParts>;
  static std::atomic<size_t> configured[64] = {};  // per instantiation, per device: largest size set so far
  int st = configure_smem(kernel, smem, configured);
  if (st != TRIS_OK) return st;
  return check_cuda(launch_kernel(kernel, dim3(ceil_div(args.out_features, kDecOut * dec_groups(P, KS)), args.num_segments, args.row_split * col_split), dim3(32 * dec_warps(P, KS)),
                                  smem, stream, pdl, col_split, args),
                    "grouped_decode_kernel launch");
}

template <int NT, int MODE>
static int dispatch_split(const TiledArgs& args, cudaStream_t stream, bool pdl) {
  // Fewer than 13 warps per SM: split the columns, as far as there are columns to split.  Of the wider tiles 20 warps fit an SM instead of 28:
  // fewer than 10 (1024 warps of 8 experts x 4096 x 256 in halves and not in quarters: blocks of 24, 40, 64 and 80 tokens 50.4 / 49.3, 59.5 / 56.1,
  // 61.4 / 58.1, 68.0 / 63.7 us).  With more than 256 columns, 14: 32 segments of 64 experts x 320 34.2 / 35.4 us.
  const long long warps = decode_warps(args, MODE) * args.row_split, split = (args.rank > 256 ? 14 : NT >= 3 ? 10 : 13) * sm_count();
  const int slices = ceil_div(args.rank, kSliceCols), groups = ceil_div(args.rank, kDecCols), want = (args.row_split > 1 ? 10 : 14) * sm_count();
  // Many columns: over the CTAs of a cluster too, by 256 columns or more each, up to 14 warps per SM (10 with shared passes).  us at 8 rows, eight warps to
  // 32 outputs in one CTA / this: 4096 x 4096 18.6 / 11.2, pair of 1024 x 4096 25.8 / 8.4, pair of 2048 x 2048 14.4 / 8.1, 512 x 1024 6.2 /
  // 4.6, 256 x 8192 33.9 / 8.2 (clusters of 1, 2, 4 and 8 CTAs in an earlier form: 4096 x 4096 24.5, 15.7, 12.0, 13.8; pair of 2048 x 2048
  // 18.1, 11.5, 8.6, 12.0).  With 512 columns two CTAs are no faster than one (2048 x 512, 8 and 24 rows 5.0 / 5.0, 6.6 / 7.5).
  // Rows that are ready before the kernel ahead has ended: that variant too, as a cluster of one at least, so that the others need not look.
  if (warps * 8 <= want && (groups >= 4 || args.rows_ready)) {
    int parts = 1;
    while (parts < 8 && warps * 8 * parts <= want && groups >= 2 * parts && groups >= 4) parts *= 2;
    return launch_decode<NT, MODE, 4, true>(args, stream, pdl, parts);
  }
  if (warps * 2 < split && slices >= 4) return launch_decode<NT, MODE, 4>(args, stream, pdl);
  if (warps < split && slices >= 4) return launch_decode<NT, MODE, 2>(args, stream, pdl);
  return launch_decode<NT, MODE, 1>(args, stream, pdl);
}

template <int MODE>
static int dispatch_decode(const TiledArgs& args, int rows, cudaStream_t stream, bool pdl) {
  if (rows <= 8) return dispatch_split<1, MODE>(args, stream, pdl);
  if (rows <= 16) return dispatch_split<2, MODE>(args, stream, pdl);
  if (rows <= 24) return dispatch_split<3, MODE>(args, stream, pdl);
  return dispatch_split<4, MODE>(args, stream, pdl);
}

int launch_grouped_decode(const TiledArgs& args, int mode, int rows, cudaStream_t stream, bool pdl) {
  if (mode == MODE_SINGLE) return dispatch_decode<MODE_SINGLE>(args, rows, stream, pdl);
  if (mode == MODE_DUAL_SILU) return dispatch_decode<MODE_DUAL_SILU>(args, rows, stream, pdl);
  return dispatch_decode<MODE_DUAL_STORE>(args, rows, stream, pdl);
}

}  // namespace tr
}  // namespace tris
