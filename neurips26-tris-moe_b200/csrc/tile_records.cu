// Builder of the tile-major records described in tile_records.cuh: a plan pass that finds the record size of a
// projection (largest salient step and row-scale slot counts over its experts), and a fill pass that decodes the
// grouping bits (Golomb-Rice streams or the sparse bitmap) and gathers the E-stacked payload tensors (QL:1512-1636 of the
// TriS-MoE tree).  Runs once per projection when a payload is prepared, and in streaming mode once per layer and pass for
// the experts that were paged in, so that they too run on the record kernels.
#include <algorithm>

#include "compact3_tile.cuh"
#include "tile_records.cuh"

namespace tris {
namespace tr {

struct BuildDims {
  int pr, nkb, nob, nblk, tiles, chunks;
};
__host__ __device__ inline BuildDims build_dims(const TrisProjView& v) {
  BuildDims d;
  d.pr = (v.rank + 31) / 32;
  d.nkb = (d.pr + 1) / 2;
  d.nob = (v.out_features + 63) / 64;
  d.nblk = d.nkb * d.nob;
  d.tiles = tiles_per_expert(v.out_features);
  d.chunks = num_chunks(v.rank);
  return d;
}
// info[1] / info[2] collect the largest slot / step counts; one thread per (expert, chunk)
__global__ void plan_records_kernel(TrisProjView v, unsigned long long* info) {
  const BuildDims d = build_dims(v);
  const int total = v.num_experts * d.chunks;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const size_t first = static_cast<size_t>(idx / d.chunks) * d.pr;
    const ChunkPlan plan = plan_chunk(v.c_map + first, v.packed_row_group ? v.packed_row_group + first : nullptr, d.pr, idx % d.chunks * kChunkRows, v.rank);
    atomicMax(&info[1], static_cast<unsigned long long>(plan.num_slots));
    atomicMax(&info[2], static_cast<unsigned long long>(plan.num_steps));
  }
}
// info: {0, slots, steps, 0} -> {total bytes, record bytes, steps, slots}; desc[i] = {offset / 16, bytes}
__global__ void describe_records_kernel(TrisProjView v, uint2* desc, int total, int64_t* info) {
  __shared__ int rec;
  if (threadIdx.x == 0) {
    const int slots = static_cast<int>(info[1]), steps = static_cast<int>(info[2]);
    rec = record_bytes(v.rank, steps, slots);
    info[0] = static_cast<int64_t>(total) * rec;
    info[1] = rec;
    info[2] = steps;
    info[3] = slots;
  }
  __syncthreads();
  if (desc == nullptr) return;
  for (int i = threadIdx.x; i < total; i += blockDim.x)
    desc[i] = make_uint2(static_cast<uint32_t>((static_cast<int64_t>(i) * rec) >> 4), static_cast<uint32_t>(rec));
  if (threadIdx.x == 0) desc[total] = make_uint2(kColMagic, 0u);
}

__device__ __forceinline__ uint32_t half_of_pack(unsigned long long pack, int which) {
  return static_cast<uint32_t>(pack >> (16 * which)) & 0xFFFFu;
}

// Where the records of a projection come from and go to.  Without expert_ids every expert's record lies at its own place; with them
// (streaming) record s is that of segment s, whose paged tensors lie in staging slot s.
struct BuildArgs {
  TrisProjView proj[2];
  uint8_t* records[2];
  uint8_t* cols[2];
  int32_t max_steps[2], max_slots[2];
  const int32_t* expert_ids;
  const int32_t* num_segments_dev;
  int32_t num_segments;
  int32_t* status;
};

// Column record of a chunk by a warp; cw, grp: the salient columns and the groups of its packed rows, cp: scales of its first column.  Salient
// columns take places in order, and a new group starts at a multiple of 16 of them (as plan_chunk deals them).  Steps and slots that the plan
// did not count are left out, so that the record's readers stay inside it.  Returns whether there were any.
__device__ __forceinline__ bool build_col_record(const TrisProjView& v, int p0, int rows, const uint32_t (&cw)[kChunkRows], const int (&grp)[kChunkRows],
                                                 const unsigned long long* cp, int max_steps, int max_slots, int lane, uint16_t* col_of, uint8_t* rec) {
  ColHeader h = {};
  h.magic = kColMagic;
  for (int i = lane; i < kMaxSteps * 16; i += 32) col_of[i] = 0xFFFFu;
  __syncwarp();
  int at = 0, slots = 0, salient = 0;
#pragma unroll
  for (int p = 0; p < kChunkRows; ++p) {
    if (p < rows && (p == 0 || grp[p] != grp[p - 1])) {
      ++slots;
      at = (at + 15) & ~15;
    }
    h.slot_of_row[p] = static_cast<uint8_t>(min(slots, max_slots) - 1);
    const int n = __popc(cw[p]), end = at + n;
    if ((cw[p] >> lane) & 1u) col_of[at + __popc(cw[p] & ((1u << lane) - 1u))] = static_cast<uint16_t>(32 * p + lane);
#pragma unroll
    for (int s = 0; s < kMaxSteps; ++s)
      if (n > 0 && 16 * s < end && 16 * s + 16 > at) h.step_slot[s] = static_cast<uint8_t>(min(slots, max_slots) - 1);
    at = end;
    salient += n;
  }
  const int steps = (at + 15) >> 4;
  h.num_slots = static_cast<uint8_t>(min(slots, max_slots));
  h.num_steps = static_cast<uint8_t>(min(steps, max_steps));
  h.num_salient = static_cast<uint16_t>(salient);
  if (lane == 0) *reinterpret_cast<ColHeader*>(rec) = h;
  __syncwarp();
  uint2* coltab = reinterpret_cast<uint2*>(rec + kColHdrBytes);
#pragma unroll
  for (int k = 0; k < kChunkCols / 64; ++k) {  // columns 2 * pair, 2 * pair + 1 of the chunk
    const int pair = lane + 32 * k, slice = pair >> 5, word = (pair >> 3) & 3, j = (pair >> 1) & 3;
    const uint32_t taken = (pair < 16 ? cw[0] : pair < 32 ? cw[1] : pair < 48 ? cw[2] : cw[3]) >> (2 * (pair & 15));
    uint2 ns = make_uint2(0u, 0u);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int c = 2 * pair + b;
      if (32 * p0 + c >= v.rank || ((taken >> b) & 1u)) continue;
      const unsigned long long pack = cp[c];
      ns.x |= half_of_pack(pack, 2) << (16 * b);
      ns.y |= half_of_pack(pack, 3) << (16 * b);
    }
    coltab[((slice * 4 + j) * 4 + word) * 2 + (pair & 1)] = ns;
  }
  for (int i = lane; i < max_steps * 8; i += 32) {
    const int step = i >> 3, pair = i & 7;
    uint8_t* ent = rec + kColHdrBytes + kColTabBytes + step * kColStepBytes;
    uint2 c = make_uint2(0u, 0u);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const unsigned col = col_of[step * 16 + 2 * pair + b];
      // an unused position names column 0 with scales of zero
      reinterpret_cast<uint16_t*>(ent + 64)[2 * pair + b] = static_cast<uint16_t>(col == 0xFFFFu ? 0u : col);
      if (col == 0xFFFFu) continue;
      const unsigned long long pack = cp[col];
      c.x |= half_of_pack(pack, 0) << (16 * b);
      c.y |= half_of_pack(pack, 1) << (16 * b);
    }
    reinterpret_cast<uint2*>(ent)[pair] = c;
  }
  return steps > max_steps || slots > max_slots;
}

// Bytes 3, 2 of the result: bits 0, 2 .. 14 and 1, 3 .. 15 of v, the first one on top; bytes 1, 0: those of the upper half.
__device__ __forceinline__ uint32_t split_reversed(uint32_t v) {
  v = __brev(v);
  uint32_t t = (v ^ (v >> 1)) & 0x22222222u;
  v ^= t ^ (t << 1);
  t = (v ^ (v >> 2)) & 0x0C0C0C0Cu;
  v ^= t ^ (t << 2);
  t = (v ^ (v >> 4)) & 0x00F000F0u;
  return v ^ t ^ (t << 4);
}
// The two code words of a packed row (32 columns) from its sign and second bits, in the order the unpack reads them.
__device__ __forceinline__ uint2 code_words(uint32_t sign, uint32_t second) {
  const uint32_t a = split_reversed(~sign), b = split_reversed(second);
  return make_uint2(prmt(a, b, 0x2637u), prmt(a, b, 0x0415u));
}

// 32 bits of a stream of rows of words, `stride` apart, from bit `first` on.
__device__ __forceinline__ uint32_t stream_bits(const uint32_t* words, int rows, int stride, int first) {
  const int q = first >> 5;
  const uint32_t lo = q < rows ? words[static_cast<size_t>(q) * stride] : 0u, hi = q + 1 < rows ? words[static_cast<size_t>(q + 1) * stride] : 0u;
  return __funnelshift_r(lo, hi, first & 31);
}

// grid (items, experts or segments, projections), 128 threads.  An item is an output tile and a pair of chunks, a thread an output of it; or,
// after those, the column records of four chunks, a warp each.  Every load is asked for before the first store, in three dependent rounds (segment,
// tables, planes): in the order of use they took turns with the stores, which may alias them for all the compiler knows.  us for 102 experts
// of 2048 x 256: 25 in that order, 30 with four outputs to a lane (fewer instructions, too few warps), 24 in this one.
// In two phases, where only the bitmap is paged: what does not need it while it is still on its way, and then only its bits.
// The first phase is compiled for six CTAs to an SM: for seven the compiler takes 72 registers and spills some, for six it takes 64 without, and
// eight fit.  Two streamed layers of 102 experts, 16 tokens: 372.8 / 366 us called from Python, 349 / 346 replayed as a graph.
enum { BUILD_ALL = 0, BUILD_BASE = 1, BUILD_BITS = 2 };
constexpr int kBuildWarps = 4, kBuildRows = 2 * kChunkRows;  // packed rows of an item
template <int PHASE>
__global__ void __launch_bounds__(32 * kBuildWarps, PHASE == BUILD_BASE ? 6 : 7) build_tile_records_kernel(const __grid_constant__ BuildArgs args) {
  __shared__ uint16_t col_of[kBuildWarps][kMaxSteps * 16];
  __shared__ uint32_t stream[kBuildWarps][TRIS_GR_BLOCK_WORDS + 4];    // a block-GR block, with read slack
  __shared__ uint32_t plane[2][4][TRIS_GR_BLOCK_WORDS];                // decoded: [chunk][k block * 2 + out block][row parity][64]
  const TrisProjView& v = args.proj[blockIdx.z];
  const int max_steps = args.max_steps[blockIdx.z], max_slots = args.max_slots[blockIdx.z];
  const BuildDims d = build_dims(v);
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31, item = blockIdx.x, place = blockIdx.y;
  const int pairs = (d.chunks + 1) / 2;
  const bool columns = item >= d.tiles * pairs;
  const int tile = item / pairs, c0 = columns ? (item - d.tiles * pairs) * kBuildWarps + warp : 2 * (item - tile * pairs);  // first chunk
  int e = place;
  if (args.expert_ids) {
    const int live = args.num_segments_dev ? *args.num_segments_dev : args.num_segments, id = args.expert_ids[place];
    if (PHASE != BUILD_BASE && live > args.num_segments && item == 0 && place == 0 && tid == 0 && args.status) *args.status = TRIS_ERR_WORKSPACE;  // no slot for them
    if (place >= live) return;
    e = warp_uniform(id);
    if (e < 0 || e >= v.num_experts) return;
  }
  if (c0 >= d.chunks) return;
  const int at = v.expert_slot ? place : e, gmap_at = v.gmap_slot ? place : at;  // places of the paged tensors
  const int p0 = c0 * kChunkRows, rows = min(kBuildRows, d.pr - p0), o = tile * kTileOut + tid, O = v.out_features;
  const bool second = v.qweight2_sparse_prefix && v.qweight2_sparse && v.sign2_rows > 0, sparse = PHASE != BUILD_BASE && !v.use_block_gr && v.q_gmap_sparse && v.gmap_sparse_rows > 0;

  // Tables of the packed rows: lane 8 k + p loads table k of row p.
  uint32_t table = 0u;
  {
    const int p = lane & 7, k = lane >> 3;
    const size_t row = static_cast<size_t>(e) * d.pr + p0 + p, prefix = row + e;  // prefixes have one entry more
    if (p < rows) {
      if (k == 0) table = static_cast<uint32_t>(v.c_map[row]);
      if (k == 1 && v.packed_row_group) table = static_cast<uint32_t>(v.packed_row_group[row]);
      if (k == 2 && sparse) table = static_cast<uint32_t>(v.q_gmap_sparse_prefix[prefix]);
      if (k == 3 && second) table = static_cast<uint32_t>(v.qweight2_sparse_prefix[prefix]);
    }
  }
  auto valid = [&](int p) {
    const int left = v.rank - 32 * (p0 + p);
    return left >= 32 ? ~0u : (left > 0 ? (1u << left) - 1u : 0u);
  };
  uint32_t salient[kBuildRows];
  int grp[kBuildRows], rank2[kBuildRows];
#pragma unroll
  for (int p = 0; p < kBuildRows; ++p) {
    salient[p] = __shfl_sync(0xFFFFFFFFu, table, p) & valid(p);
    grp[p] = static_cast<int>(__shfl_sync(0xFFFFFFFFu, table, 8 + p));
    rank2[p] = static_cast<int>(__shfl_sync(0xFFFFFFFFu, table, 24 + p));
  }
  if (columns) {
    const uint32_t cw[kChunkRows] = {salient[0], salient[1], salient[2], salient[3]};
    const int gr[kChunkRows] = {grp[0], grp[1], grp[2], grp[3]};
    const bool more = build_col_record(v, p0, min(kChunkRows, rows), cw, gr, reinterpret_cast<const unsigned long long*>(v.col_pack3) + static_cast<size_t>(at) * v.rank + 32 * p0,
                                       max_steps, max_slots, lane, col_of[warp], args.cols[blockIdx.z] + static_cast<size_t>(place * d.chunks + c0) * col_record_bytes(max_steps));
    if (more && lane == 0 && args.status) *args.status = TRIS_ERR_CORRUPT;  // the payload is not the one that was planned
    return;
  }

  const bool live = o < O;
  auto opens = [&](int p) { return p < rows && (p % kChunkRows == 0 || grp[p] != grp[p - 1]); };  // a row-scale slot
  const int slices = record_slices(v.rank), size = record_bytes(v.rank, max_steps, max_slots), sub_bytes = size / kSubs;
  uint8_t* rec = args.records[blockIdx.z] + static_cast<size_t>((place * d.tiles + tile) * d.chunks + c0) * static_cast<size_t>(size) + warp * sub_bytes;
  uint32_t s[kBuildRows], g[kBuildRows], run2[2];    // run2: second signs of a chunk's first 32 salient columns
  unsigned long long scales[kBuildRows];             // of the row's group, where that is a new one
  const uint32_t* signs = reinterpret_cast<const uint32_t*>(v.qweight1) + (static_cast<size_t>(at) * d.pr + p0) * O + o;
  const uint32_t* signs2 = reinterpret_cast<const uint32_t*>(v.qweight2_sparse) + static_cast<size_t>(at) * v.sign2_rows * O + o;
  const uint32_t* bitmap = reinterpret_cast<const uint32_t*>(v.q_gmap_sparse) + static_cast<size_t>(gmap_at) * v.gmap_sparse_rows * O + o;
  const auto codes = [&](int c, int sl) { return reinterpret_cast<uint4*>(rec + static_cast<size_t>(c) * static_cast<size_t>(size) + sl * kSliceBytes) + lane; };
  uint4 base[2][2];  // the code words that the first phase wrote
  if constexpr (PHASE == BUILD_BITS) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int sl = 0; sl < 2; ++sl)
        if (c * kChunkRows < rows && sl < slices) base[c][sl] = *codes(c, sl);
  }
  const unsigned long long* row_scales = reinterpret_cast<const unsigned long long*>(v.row_pack3) + (static_cast<size_t>(at) * O + o) * v.num_groups;
#pragma unroll
  for (int p = 0; p < kBuildRows; ++p) {
    const bool there = live && p < rows;
    s[p] = PHASE != BUILD_BITS && there ? signs[static_cast<size_t>(p) * O] : 0u;
    const int first = max(0, static_cast<int>(__shfl_sync(0xFFFFFFFFu, table, 16 + p)));
    g[p] = there && sparse ? stream_bits(bitmap, v.gmap_sparse_rows, O, first) : 0u;
    scales[p] = PHASE != BUILD_BITS && live && opens(p) && grp[p] >= 0 && grp[p] < v.num_groups ? row_scales[grp[p]] : 0ull;
  }
#pragma unroll
  for (int c = 0; c < 2; ++c)
    run2[c] = PHASE != BUILD_BITS && live && second && rank2[c * kChunkRows] >= 0 && c * kChunkRows < rows ? stream_bits(signs2, v.sign2_rows, O, rank2[c * kChunkRows]) : 0u;

  if (PHASE == BUILD_ALL && v.use_block_gr) {  // per chunk two k blocks of two out blocks, a warp each (decode_block_gr_block, CU:426-479)
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
      uint32_t* out = plane[c][warp];
      for (int i = lane; i < TRIS_GR_BLOCK_WORDS; i += 32) out[i] = 0u;
      const int kb = (kChunkRows / 2) * (c0 + c) + (warp >> 1), ob = 2 * tile + (warp & 1), bi = kb * d.nob + ob;
      int count = 0, meta = 0, src = 0;
      if (kb < d.nkb && ob < d.nob) {
        const int32_t* off = v.q_gmap_gr_offsets + static_cast<size_t>(e) * (d.nblk + 1);
        src = off[bi];
        count = max(0, min(off[bi + 1] - src, TRIS_GR_BLOCK_WORDS));
        meta = v.q_gmap_gr_meta[static_cast<size_t>(e) * d.nblk + bi];
      }
      const uint32_t* words = reinterpret_cast<const uint32_t*>(v.q_gmap_gr_words) + static_cast<size_t>(at) * v.gr_max_words;
      for (int i = lane; i < TRIS_GR_BLOCK_WORDS + 4; i += 32)
        stream[warp][i] = (i < count && src + i >= 0 && src + i < v.gr_max_words) ? words[src + i] : 0u;
      __syncwarp();
      if (count > 0) {
        if (meta & TRIS_GR_META_RAW_FLAG) {
          for (int i = lane; i < count; i += 32) out[i] = stream[warp][i];
        } else {
          const int ones = min(meta >> TRIS_GR_META_ONE_COUNT_SHIFT, TRIS_GR_BLOCK_WORDS * 32);
          const int per = (ones + 31) >> 5, from = lane * per;
          if (per > 0 && from < ones) {
            const uint32_t sub = v.gr_index[(static_cast<size_t>(at) * d.nblk + bi) * 32 + lane];
            gr_decode_run(stream[warp], count, meta & TRIS_GR_META_K_MASK, min(per, ones - from), static_cast<int>(sub & 0xFFFFu),
                          static_cast<int>(sub >> 16), [&](int flat) { atomicOr(out + (flat >> 5), 1u << (flat & 31)); });
          }
        }
      }
      __syncwarp();
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < kBuildRows; ++p) {
      const int q = p % kChunkRows;
      if (live && p < rows) g[p] = plane[p / kChunkRows][(q >> 1) * 2 + (tid >> 6)][(q & 1) * 64 + (tid & 63)];
    }
  } else if (sparse) {  // the bitmap leaves the salient columns out: what lies at or above one moves up by one
#pragma unroll
    for (int p = 0; p < kBuildRows; ++p) {
#pragma unroll 1
      for (uint32_t m = salient[p]; m; m &= m - 1) g[p] += g[p] & (0u - (m & (0u - m)));
      g[p] &= valid(p) & ~salient[p];
    }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (c * kChunkRows >= rows) break;
#pragma unroll
    for (int sl = 0; sl < kChunkRows / 2; ++sl) {
      if (sl >= slices) break;
      const int p = c * kChunkRows + 2 * sl;
      const uint2 a = code_words(PHASE == BUILD_BITS ? ~0u : s[p], g[p]), b = code_words(PHASE == BUILD_BITS ? ~0u : s[p + 1], g[p + 1]);
      uint4 w = make_uint4(a.x, a.y, b.x, b.y);
      if (PHASE == BUILD_BITS) w = make_uint4(w.x | base[c][sl].x, w.y | base[c][sl].y, w.z | base[c][sl].z, w.w | base[c][sl].w);
      *codes(c, sl) = w;
    }
    if (PHASE == BUILD_BITS) continue;
    // Salient steps and row-scale slots, as plan_chunk deals them: a new group opens a slot, and the next salient column a step.
    uint8_t* tail = rec + static_cast<size_t>(c) * static_cast<size_t>(size) + slices * kSliceBytes;
    uint32_t* step_at = reinterpret_cast<uint32_t*>(tail) + lane;
    uint2* slot_at = reinterpret_cast<uint2*>(tail + max_steps * kStepBytes) + lane;
    const int first2 = rank2[c * kChunkRows];
    int steps = 0, slots = 0, fill = 16, begin2 = 0;
    uint32_t w1 = 0u;
    auto close = [&]() {  // writes step `steps` - 1: its second sign bits follow one another
      const int ahead = begin2 - first2;
      uint32_t w2 = run2[c] >> (ahead & 31);
      if (ahead > 16 && live && second && begin2 >= 0) w2 = stream_bits(signs2, v.sign2_rows, O, begin2);
      if (steps <= max_steps) step_at[(steps - 1) * kSubOut] = code_words(w1, ~(w2 & ((1u << fill) - 1u))).x;  // both bits as "negative"
      w1 = 0u;
    };
#pragma unroll
    for (int q = 0; q < kChunkRows; ++q) {
      const int p = c * kChunkRows + q;
      if (p >= rows) break;
      if (opens(p)) {
        if (fill < 16) close();
        fill = 16;
        if (slots < max_slots) slot_at[slots * kSubOut] = make_uint2(static_cast<uint32_t>(scales[p]), static_cast<uint32_t>(scales[p] >> 32));
        ++slots;
      }
      int at2 = rank2[p];
#pragma unroll 1
      for (uint32_t m = salient[p]; m; m &= m - 1, ++at2) {
        if (fill == 16) {
          fill = 0;
          ++steps;
          begin2 = at2;
        }
        w1 |= ((s[p] >> (__ffs(m) - 1)) & 1u) << fill;
        if (++fill == 16) close();
      }
    }
    if (fill < 16) close();
    for (; steps < max_steps; ++steps) step_at[steps * kSubOut] = code_words(0u, ~0u).x;
    for (; slots < max_slots; ++slots) slot_at[slots * kSubOut] = make_uint2(0u, 0u);
  }
}

// Items of a projection: tiles times pairs of chunks, and the column records.
static int build_items(const BuildDims& d) { return d.tiles * ((d.chunks + 1) / 2) + ceil_div(d.chunks, kBuildWarps); }
static int launch_build(const BuildArgs& args, int items, int places, int projections, int phase, cudaStream_t stream) {
  auto kernel = phase == BUILD_ALL ? build_tile_records_kernel<BUILD_ALL> : (phase == BUILD_BASE ? build_tile_records_kernel<BUILD_BASE> : build_tile_records_kernel<BUILD_BITS>);
  kernel<<<dim3(items, places, projections), 32 * kBuildWarps, 0, stream>>>(args);
  return check_cuda(cudaGetLastError(), "build_tile_records_kernel launch");
}

// Row-scale slots follow from the record size that the plan found (max_record_bytes of the view); 0: it is not such a size.
static int slots_of(const TrisProjView& v, int max_steps) {
  const int slots = (v.max_record_bytes - record_bytes(v.rank, max_steps, 0)) / (kSubs * kSlotBytes);
  return slots >= 1 && slots <= kChunkRows && v.max_record_bytes == record_bytes(v.rank, max_steps, slots) ? slots : 0;
}

static int validate_dims(const TrisProjView* v, const char* name) {
  TRIS_REQUIRE(v != nullptr, TRIS_ERR_INVALID_ARG, "%s: null projection view", name);
  TRIS_REQUIRE(v->num_experts > 0 && v->out_features > 0 && v->rank > 0 && v->num_groups > 0, TRIS_ERR_INVALID_ARG,
               "%s: non-positive dims", name);
  return TRIS_OK;
}
static int validate_for_records(const TrisProjView* v, const char* name, bool paged = false) {
  const int st = validate_dims(v, name);
  if (st != TRIS_OK) return st;
  if (!v->use_block_gr && paged) {
    TRIS_REQUIRE(v->gmap_sparse_rows == 0 || (v->q_gmap_sparse && v->q_gmap_sparse_prefix), TRIS_ERR_INVALID_ARG, "%s: q_gmap_sparse needs its prefix", name);
  } else {
    TRIS_REQUIRE(v->use_block_gr && v->q_gmap_gr_words && v->q_gmap_gr_offsets && v->q_gmap_gr_meta, TRIS_ERR_UNSUPPORTED,
                 "%s: tile records need a block-GR payload", name);
    TRIS_REQUIRE(v->gr_index != nullptr && v->gr_substreams == 32, TRIS_ERR_INVALID_ARG,
                 "%s: needs the 32-way sub-stream index (tris_block_gr_build_index)", name);
  }
  TRIS_REQUIRE(v->qweight1 && v->c_map && v->col_pack3 && v->row_pack3, TRIS_ERR_INVALID_ARG,
               "%s: qweight1/c_map/col_pack3/row_pack3 must be set", name);
  TRIS_REQUIRE(v->packed_row_group != nullptr || v->num_groups == 1, TRIS_ERR_INVALID_ARG,
               "%s: packed_row_group missing (call tris_build_row_groups)", name);
  TRIS_REQUIRE(paged || (!v->expert_slot && !v->gmap_slot), TRIS_ERR_UNSUPPORTED, "%s: paged payloads have no tile records", name);
  return TRIS_OK;
}

}  // namespace tr

int build_paged_records(const TrisProjView* staged, const TrisProjView* records, int projections, const TrisRouteView* route, int capacity, bool paged,
                        cudaStream_t stream) {
  using namespace tr;
  BuildArgs args{};
  int items = 0;
  bool in_two = true;  // only the bitmap is paged
  for (int i = 0; i < projections; ++i) in_two = in_two && !staged[i].use_block_gr && staged[i].gmap_slot && !staged[i].expert_slot;
  if (!paged && !in_two) return TRIS_OK;
  const int phase = !in_two ? BUILD_ALL : (paged ? BUILD_BITS : BUILD_BASE);
  for (int i = 0; i < projections; ++i) {
    const int st = validate_for_records(staged + i, "paged tile records", true);
    if (st != TRIS_OK) return st;
    const TrisProjView& r = records[i];
    TRIS_REQUIRE(r.rank == staged[i].rank && r.out_features == staged[i].out_features && r.num_experts == capacity && proj_has_tile_records(r) &&
                     r.max_sal_words >= 0 && r.max_sal_words <= kMaxSteps && r.col_record_bytes == col_record_bytes(r.max_sal_words) && slots_of(r, r.max_sal_words) > 0,
                 TRIS_ERR_INVALID_ARG, "paged tile records: the record view does not belong to the projection");
    TRIS_REQUIRE(((reinterpret_cast<uintptr_t>(r.tile_records) | reinterpret_cast<uintptr_t>(r.col_records)) & 15u) == 0, TRIS_ERR_INVALID_ARG,
                 "paged tile records: buffers must be 16-byte aligned");
    args.proj[i] = staged[i];
    args.records[i] = static_cast<uint8_t*>(const_cast<void*>(r.tile_records));
    args.cols[i] = static_cast<uint8_t*>(const_cast<void*>(r.col_records));
    args.max_steps[i] = r.max_sal_words;
    args.max_slots[i] = slots_of(r, r.max_sal_words);
    const BuildDims d = build_dims(r);
    items = std::max(items, build_items(d) - (phase == BUILD_BITS ? ceil_div(d.chunks, kBuildWarps) : 0));
  }
  args.expert_ids = route->expert_ids;
  args.num_segments_dev = route->num_segments_dev;
  args.num_segments = std::min(route->num_segments, capacity);
  args.status = route->status_dev;
  return launch_build(args, items, args.num_segments, projections, phase, stream);
}

}  // namespace tris

using namespace tris;
using namespace tris::tr;

extern "C" int64_t tris_tile_record_count(const TrisProjView* proj) {
  if (proj == nullptr || proj->num_experts <= 0 || proj->out_features <= 0 || proj->rank <= 0) return 0;
  const BuildDims d = build_dims(*proj);
  return static_cast<int64_t>(proj->num_experts) * d.tiles * d.chunks;
}

extern "C" int64_t tris_col_record_bytes(const TrisProjView* proj, int32_t max_sal_words) {
  if (proj == nullptr || max_sal_words < 0 || max_sal_words > kMaxSteps) return 0;
  const BuildDims d = build_dims(*proj);
  return static_cast<int64_t>(proj->num_experts) * d.chunks * col_record_bytes(max_sal_words);
}

extern "C" int tris_tile_records_plan(const TrisProjView* proj, uint32_t* desc_out, int64_t* info_out, void* stream) {
  int st = validate_for_records(proj, "tris_tile_records_plan");
  if (st != TRIS_OK) return st;
  TRIS_REQUIRE(desc_out && info_out, TRIS_ERR_INVALID_ARG, "tris_tile_records_plan: null output");
  const int64_t total = tris_tile_record_count(proj);
  TRIS_REQUIRE(total > 0 && total < (1ll << 30), TRIS_ERR_UNSUPPORTED, "tris_tile_records_plan: %lld records", static_cast<long long>(total));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  TRIS_CUDA(cudaMemsetAsync(info_out, 0, 4 * sizeof(int64_t), s));
  const int threads = 128, work = proj->num_experts * build_dims(*proj).chunks;
  plan_records_kernel<<<std::min((work + threads - 1) / threads, 4096), threads, 0, s>>>(*proj, reinterpret_cast<unsigned long long*>(info_out));
  TRIS_CUDA(cudaGetLastError());
  describe_records_kernel<<<1, 1024, 0, s>>>(*proj, reinterpret_cast<uint2*>(desc_out), static_cast<int>(total), info_out);
  return check_cuda(cudaGetLastError(), "tile record plan kernels");
}

extern "C" int tris_tile_records_build(const TrisProjView* proj, const uint32_t* desc, void* records_out,
                                       void* col_records_out, int32_t max_sal_words, void* stream) {
  int st = validate_for_records(proj, "tris_tile_records_build");
  if (st != TRIS_OK) return st;
  TRIS_REQUIRE(desc && records_out && col_records_out, TRIS_ERR_INVALID_ARG, "tris_tile_records_build: null pointer");
  TRIS_REQUIRE(max_sal_words >= 0 && max_sal_words <= kMaxSteps, TRIS_ERR_INVALID_ARG, "tris_tile_records_build: max_sal_words=%d",
               max_sal_words);
  TRIS_REQUIRE((reinterpret_cast<uintptr_t>(records_out) & 15u) == 0 && (reinterpret_cast<uintptr_t>(col_records_out) & 15u) == 0,
               TRIS_ERR_INVALID_ARG, "tris_tile_records_build: record buffers must be 16-byte aligned");
  const BuildDims d = build_dims(*proj);
  BuildArgs args{};
  args.proj[0] = *proj;
  args.records[0] = static_cast<uint8_t*>(records_out);
  args.cols[0] = static_cast<uint8_t*>(col_records_out);
  args.max_steps[0] = max_sal_words;
  args.max_slots[0] = slots_of(*proj, max_sal_words);
  TRIS_REQUIRE(args.max_slots[0] > 0, TRIS_ERR_INVALID_ARG, "tris_tile_records_build: max_record_bytes=%d of the view is not the plan's record size",
               proj->max_record_bytes);
  return launch_build(args, build_items(d), proj->num_experts, 1, BUILD_ALL, static_cast<cudaStream_t>(stream));
}

extern "C" int tris_paged_records_plan(const TrisProjView* proj, int64_t* info_out, void* stream) {
  int st = validate_dims(proj, "tris_paged_records_plan");
  if (st != TRIS_OK) return st;
  TRIS_REQUIRE(info_out && proj->c_map && (proj->packed_row_group || proj->num_groups == 1), TRIS_ERR_INVALID_ARG, "tris_paged_records_plan: null pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  TRIS_CUDA(cudaMemsetAsync(info_out, 0, 4 * sizeof(int64_t), s));
  const int threads = 128, work = proj->num_experts * build_dims(*proj).chunks;
  plan_records_kernel<<<std::min((work + threads - 1) / threads, 4096), threads, 0, s>>>(*proj, reinterpret_cast<unsigned long long*>(info_out));
  TRIS_CUDA(cudaGetLastError());
  describe_records_kernel<<<1, 32, 0, s>>>(*proj, nullptr, build_dims(*proj).tiles * build_dims(*proj).chunks, info_out);
  return check_cuda(cudaGetLastError(), "paged record plan kernels");
}
