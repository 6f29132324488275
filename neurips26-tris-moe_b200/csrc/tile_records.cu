// Load-time builder of the tile-major records described in tile_records.cuh: a plan pass that finds
// the record size of a projection (largest salient step and row-scale slot counts over its experts),
// and a fill pass that decodes the Golomb-Rice streams and gathers the E-stacked payload tensors
// (QL:1512-1636 of the TriS-MoE tree).  Runs once per projection when a payload is prepared; nothing
// here is on the per-token path.
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
__device__ __forceinline__ void plan_of(const TrisProjView& v, const BuildDims& d, int e, int chunk, ChunkPlan& plan, uint16_t* cols) {
  plan_chunk(v.c_map + static_cast<size_t>(e) * d.pr, v.packed_row_group ? v.packed_row_group + static_cast<size_t>(e) * d.pr : nullptr,
             d.pr, chunk * kChunkRows, v.rank, plan, cols);
}

// info[1] / info[2] collect the largest slot / step counts; one thread per (expert, chunk)
__global__ void plan_records_kernel(TrisProjView v, unsigned long long* info) {
  const BuildDims d = build_dims(v);
  const int total = v.num_experts * d.chunks;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    ChunkPlan plan;
    plan_of(v, d, idx / d.chunks, idx % d.chunks, plan, nullptr);
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
  for (int i = threadIdx.x; i < total; i += blockDim.x)
    desc[i] = make_uint2(static_cast<uint32_t>((static_cast<int64_t>(i) * rec) >> 4), static_cast<uint32_t>(rec));
  if (threadIdx.x == 0) desc[total] = make_uint2(kColMagic, 0u);
}

__device__ __forceinline__ uint32_t half_of_pack(unsigned long long pack, int which) {
  return static_cast<uint32_t>(pack >> (16 * which)) & 0xFFFFu;
}

// grid (chunks, E), 128 threads
__global__ void __launch_bounds__(128) build_col_records_kernel(TrisProjView v, uint8_t* col_records, int max_steps) {
  __shared__ ChunkPlan plan;
  __shared__ uint16_t col_of_slot[kMaxSteps * 16];
  const BuildDims d = build_dims(v);
  const int chunk = blockIdx.x, e = blockIdx.y, p0 = chunk * kChunkRows;
  uint8_t* rec = col_records + (static_cast<size_t>(e) * d.chunks + chunk) * col_record_bytes(max_steps);
  const int32_t* cmap = v.c_map + static_cast<size_t>(e) * d.pr;
  const unsigned long long* cp = reinterpret_cast<const unsigned long long*>(v.col_pack3) + static_cast<size_t>(e) * v.rank;
  if (threadIdx.x == 0) {
    plan_of(v, d, e, chunk, plan, col_of_slot);
    ColHeader h = {};
    h.magic = kColMagic;
    h.num_slots = static_cast<uint8_t>(plan.num_slots);
    h.num_steps = static_cast<uint8_t>(plan.num_steps);
    h.num_salient = static_cast<uint16_t>(plan.num_salient);
    for (int p = 0; p < kChunkRows; ++p) h.slot_of_row[p] = plan.slot_of_row[p];
    for (int s = 0; s < kMaxSteps; ++s) h.step_slot[s] = plan.step_slot[s];
    *reinterpret_cast<ColHeader*>(rec) = h;
  }
  __syncthreads();
  uint2* coltab = reinterpret_cast<uint2*>(rec + kColHdrBytes);
  if (threadIdx.x < kChunkCols / 2) {
    const int pair = threadIdx.x;  // columns 2 * pair, 2 * pair + 1 of the chunk
    uint2 ns = make_uint2(0u, 0u);
    for (int h = 0; h < 2; ++h) {
      const int c = 32 * p0 + 2 * pair + h;
      if (c >= v.rank || ((static_cast<uint32_t>(cmap[c >> 5]) >> (c & 31)) & 1u)) continue;
      ns.x |= half_of_pack(cp[c], 2) << (16 * h);
      ns.y |= half_of_pack(cp[c], 3) << (16 * h);
    }
    const int slice = pair >> 5, word = (pair >> 3) & 3, j = (pair >> 1) & 3;
    coltab[((slice * 4 + j) * 4 + word) * 2 + (pair & 1)] = ns;
  }
  for (int i = threadIdx.x; i < max_steps * 8; i += blockDim.x) {
    const int step = i >> 3, pair = i & 7;
    uint8_t* ent = rec + kColHdrBytes + kColTabBytes + step * kColStepBytes;
    uint2 c = make_uint2(0u, 0u);
    for (int h = 0; h < 2; ++h) {
      const unsigned col = col_of_slot[step * 16 + 2 * pair + h];
      // an unused position names column 0 with scales of zero
      reinterpret_cast<uint16_t*>(ent + 64)[2 * pair + h] = static_cast<uint16_t>(col == 0xFFFFu ? 0u : col);
      if (col == 0xFFFFu) continue;
      const unsigned long long pack = cp[32 * p0 + col];
      c.x |= half_of_pack(pack, 0) << (16 * h);
      c.y |= half_of_pack(pack, 1) << (16 * h);
    }
    reinterpret_cast<uint2*>(ent)[pair] = c;
  }
}

// Places 16 sign / second bits in the order the unpack reads them (bits i: 0..15 = column).
__device__ __forceinline__ uint32_t code_word(uint32_t sign16, uint32_t second16) {
  uint32_t w = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    w |= ((~sign16 >> (2 * i)) & 1u) << (15 - i);
    w |= ((~sign16 >> (2 * i + 1)) & 1u) << (31 - i);
    w |= ((second16 >> (2 * i)) & 1u) << (7 - i);
    w |= ((second16 >> (2 * i + 1)) & 1u) << (23 - i);
  }
  return w;
}

// grid (tiles * chunks, E), 128 threads
__global__ void __launch_bounds__(128) build_tile_records_kernel(TrisProjView v, uint8_t* records, int max_steps, int max_slots) {
  __shared__ ChunkPlan plan;
  __shared__ uint16_t col_of_slot[kMaxSteps * 16];
  __shared__ int slot_group[kChunkRows];
  __shared__ uint32_t stream[4][TRIS_GR_BLOCK_WORDS + 4];  // one block-GR block per warp, with read slack
  __shared__ uint32_t plane[4][TRIS_GR_BLOCK_WORDS];       // decoded: [block = k block * 2 + out block][row parity][64]
  const BuildDims d = build_dims(v);
  const int chunk = blockIdx.x % d.chunks, tile = blockIdx.x / d.chunks, e = blockIdx.y;
  const int p0 = chunk * kChunkRows, o0 = tile * kTileOut;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* rec = records + static_cast<size_t>((e * d.tiles + tile) * d.chunks + chunk) * record_bytes(v.rank, max_steps, max_slots);
  const int32_t* cmap = v.c_map + static_cast<size_t>(e) * d.pr;
  const int32_t* groups = v.packed_row_group ? v.packed_row_group + static_cast<size_t>(e) * d.pr : nullptr;
  if (tid < kChunkRows) slot_group[tid] = -1;
  __syncthreads();
  if (tid == 0) {
    plan_of(v, d, e, chunk, plan, col_of_slot);
    for (int p = 0; p < kChunkRows; ++p)
      if (p0 + p < d.pr) slot_group[plan.slot_of_row[p]] = groups ? groups[p0 + p] : 0;
  }
  // block-GR: warp w decodes k block w / 2 of out block w % 2 (decode_block_gr_block, CU:426-479)
  for (int i = lane; i < TRIS_GR_BLOCK_WORDS; i += 32) plane[warp][i] = 0u;
  const int kb = (kChunkRows / 2) * chunk + (warp >> 1), ob = 2 * tile + (warp & 1);
  int count = 0, meta = 0, src = 0;
  const int bi = kb * d.nob + ob;
  if (kb < d.nkb && ob < d.nob) {
    const int32_t* off = v.q_gmap_gr_offsets + static_cast<size_t>(e) * (d.nblk + 1);
    src = off[bi];
    count = max(0, min(off[bi + 1] - src, TRIS_GR_BLOCK_WORDS));
    meta = v.q_gmap_gr_meta[static_cast<size_t>(e) * d.nblk + bi];
  }
  const uint32_t* words = reinterpret_cast<const uint32_t*>(v.q_gmap_gr_words) + static_cast<size_t>(e) * v.gr_max_words;
  for (int i = lane; i < TRIS_GR_BLOCK_WORDS + 4; i += 32)
    stream[warp][i] = (i < count && src + i >= 0 && src + i < v.gr_max_words) ? words[src + i] : 0u;
  __syncwarp();
  if (count > 0) {
    if (meta & TRIS_GR_META_RAW_FLAG) {
      for (int i = lane; i < count; i += 32) plane[warp][i] = stream[warp][i];
    } else {
      const int ones = min(meta >> TRIS_GR_META_ONE_COUNT_SHIFT, TRIS_GR_BLOCK_WORDS * 32);
      const int per = (ones + 31) >> 5, first = lane * per;
      if (per > 0 && first < ones) {
        const uint32_t at = v.gr_index[(static_cast<size_t>(e) * d.nblk + bi) * 32 + lane];
        uint32_t* out = plane[warp];
        gr_decode_run(stream[warp], count, meta & TRIS_GR_META_K_MASK, min(per, ones - first), static_cast<int>(at & 0xFFFFu),
                      static_cast<int>(at >> 16), [&](int flat) { atomicOr(out + (flat >> 5), 1u << (flat & 31)); });
      }
    }
  }
  __syncthreads();
  const uint32_t* qw1 = reinterpret_cast<const uint32_t*>(v.qweight1) + static_cast<size_t>(e) * d.pr * v.out_features;
  const int32_t* pre2 = v.qweight2_sparse_prefix ? v.qweight2_sparse_prefix + static_cast<size_t>(e) * (d.pr + 1) : nullptr;
  const uint32_t* qw2 = reinterpret_cast<const uint32_t*>(v.qweight2_sparse) + static_cast<size_t>(e) * v.sign2_rows * v.out_features;
  auto sign2_bit = [&](int pg, int bit, int o) -> uint32_t {  // salient column 32 * pg + bit
    if (!pre2 || !v.qweight2_sparse || v.sign2_rows <= 0) return 0u;
    const int r2 = pre2[pg] + __popc(static_cast<uint32_t>(cmap[pg]) & ((1u << bit) - 1u));
    if (r2 < 0 || (r2 >> 5) >= v.sign2_rows) return 0u;
    return (qw2[static_cast<size_t>(r2 >> 5) * v.out_features + o] >> (r2 & 31)) & 1u;
  };
  const int slices = record_slices(v.rank), sub_bytes = record_bytes(v.rank, max_steps, max_slots) / kSubs;
  // codes: item = (packed row, output); two code words each
  for (int i = tid; i < slices * 2 * kTileOut; i += blockDim.x) {
    const int p = i / kTileOut, ol = i % kTileOut, o = o0 + ol, pg = p0 + p;
    uint32_t s = 0u, g = 0u;
    if (pg < d.pr && o < v.out_features) {
      s = qw1[static_cast<size_t>(pg) * v.out_features + o];
      g = plane[(p >> 1) * 2 + (ol >> 6)][(p & 1) * 64 + (ol & 63)];
    }
    uint32_t* dst = reinterpret_cast<uint32_t*>(rec + (ol >> 5) * sub_bytes + (p >> 1) * kSliceBytes + (ol & 31) * 16) + (p & 1) * 2;
    dst[0] = code_word(s & 0xFFFFu, g & 0xFFFFu);
    dst[1] = code_word(s >> 16, g >> 16);
  }
  // salient steps
  for (int i = tid; i < max_steps * kTileOut; i += blockDim.x) {
    const int step = i / kTileOut, ol = i % kTileOut, o = o0 + ol;
    uint32_t w1 = 0u, w2 = 0u;
    if (step < plan.num_steps && o < v.out_features) {
      for (int j = 0; j < 16; ++j) {
        const unsigned col = col_of_slot[step * 16 + j];
        if (col == 0xFFFFu) continue;
        const int pg = p0 + static_cast<int>(col >> 5), bit = col & 31;
        w1 |= ((qw1[static_cast<size_t>(pg) * v.out_features + o] >> bit) & 1u) << j;
        w2 |= sign2_bit(pg, bit, o) << j;
      }
    }
    reinterpret_cast<uint32_t*>(rec + (ol >> 5) * sub_bytes + slices * kSliceBytes + step * kStepBytes)[ol & 31] =
        code_word(w1, ~w2);  // both bits as "negative"
  }
  // row scales
  for (int i = tid; i < max_slots * kTileOut; i += blockDim.x) {
    const int slot = i / kTileOut, ol = i % kTileOut, o = o0 + ol;
    const int grp = slot < kChunkRows ? slot_group[slot] : -1;
    unsigned long long w = 0ull;
    if (o < v.out_features && grp >= 0 && grp < v.num_groups)
      w = static_cast<unsigned long long>(v.row_pack3[(static_cast<size_t>(e) * v.out_features + o) * v.num_groups + grp]);
    reinterpret_cast<uint2*>(rec + (ol >> 5) * sub_bytes + slices * kSliceBytes + max_steps * kStepBytes + slot * kSlotBytes)[ol & 31] =
        make_uint2(static_cast<uint32_t>(w), static_cast<uint32_t>(w >> 32));
  }
}

static int validate_for_records(const TrisProjView* v, const char* name) {
  TRIS_REQUIRE(v != nullptr, TRIS_ERR_INVALID_ARG, "%s: null projection view", name);
  TRIS_REQUIRE(v->num_experts > 0 && v->out_features > 0 && v->rank > 0 && v->num_groups > 0, TRIS_ERR_INVALID_ARG,
               "%s: non-positive dims", name);
  TRIS_REQUIRE(v->use_block_gr && v->q_gmap_gr_words && v->q_gmap_gr_offsets && v->q_gmap_gr_meta, TRIS_ERR_UNSUPPORTED,
               "%s: tile records need a block-GR payload", name);
  TRIS_REQUIRE(v->gr_index != nullptr && v->gr_substreams == 32, TRIS_ERR_INVALID_ARG,
               "%s: needs the 32-way sub-stream index (tris_block_gr_build_index)", name);
  TRIS_REQUIRE(v->qweight1 && v->c_map && v->col_pack3 && v->row_pack3, TRIS_ERR_INVALID_ARG,
               "%s: qweight1/c_map/col_pack3/row_pack3 must be set", name);
  TRIS_REQUIRE(v->packed_row_group != nullptr || v->num_groups == 1, TRIS_ERR_INVALID_ARG,
               "%s: packed_row_group missing (call tris_build_row_groups)", name);
  TRIS_REQUIRE(!v->expert_slot && !v->gmap_slot, TRIS_ERR_UNSUPPORTED, "%s: paged payloads have no tile records", name);
  return TRIS_OK;
}

}  // namespace tr
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
  // the row-scale slots follow from the record size the plan found (max_record_bytes of the view)
  const int slots = (proj->max_record_bytes - record_bytes(proj->rank, max_sal_words, 0)) / (kSubs * kSlotBytes);
  TRIS_REQUIRE(slots >= 1 && slots <= kChunkRows && proj->max_record_bytes == record_bytes(proj->rank, max_sal_words, slots),
               TRIS_ERR_INVALID_ARG, "tris_tile_records_build: max_record_bytes=%d of the view is not the plan's record size",
               proj->max_record_bytes);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  build_col_records_kernel<<<dim3(d.chunks, proj->num_experts), 128, 0, s>>>(*proj, static_cast<uint8_t*>(col_records_out), max_sal_words);
  TRIS_CUDA(cudaGetLastError());
  build_tile_records_kernel<<<dim3(d.tiles * d.chunks, proj->num_experts), 128, 0, s>>>(*proj, static_cast<uint8_t*>(records_out),
                                                                                        max_sal_words, slots);
  return check_cuda(cudaGetLastError(), "tile record build kernels");
}
