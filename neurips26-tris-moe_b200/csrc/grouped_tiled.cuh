// What the tile-record kernels share: launch arguments, result stores, host helpers.
// grouped_decode.cu: few rows per segment, many small CTAs; grouped_tiled.cu: wide passes, persistent
// warp-specialised CTAs; grouped_wide.cu: the same with a segment's weights kept in shared memory.
#pragma once
#include <algorithm>
#include <atomic>

#include "tile_records.cuh"
#include "umma.cuh"

namespace tris {
namespace tr {

enum { MODE_SINGLE = 0, MODE_DUAL_STORE = 1, MODE_DUAL_SILU = 2 };

constexpr int kACols = kSliceCols / 2;  // TMEM columns of one 64-column slice of weights

struct TiledArgs {
  TrisProjView proj[2];
  const __half* hidden[2];
  __half* out[2];
  const int32_t* expert_ids;
  const int32_t* segment_offsets;
  const int32_t* num_segments_dev;
  const int32_t* row_gather;
  const int32_t* out_scatter;
  int32_t* status;
  int32_t num_segments;
  int32_t num_rows;
  int32_t rank, out_features, num_experts;  // the same for both projections
  int32_t tiles, chunks, units_x, row_split;
  int32_t col_split, pass_chunks;  // parts of the chunks that different CTAs take; chunks of the longest part
  int32_t max_steps;            // salient steps a record of either projection can have
  int32_t max_sub_bytes;        // larger sub-record of the two projections
  int32_t hidden_mode;          // column order of the activation rows (TRIS_OUT_F16 / _PAIR_INTERLEAVED / _LANE_ORDER)
  int32_t hidden_stride;        // halves between activation rows
  int32_t hidden_vec;           // rows can be copied in 16-byte pieces as they are
  int32_t hidden_perm;          // rows in a permuted order that can be read word by word
  int32_t num_sets;             // 2 when the two projections read different activation rows
  int32_t weights_before_wait;  // route arrays were final before the predecessor kernel started
  int32_t stages;               // ring depth, 2 .. kMaxStages
  int32_t reuse;                // the chunks of a pass fit the ring: staged once for all tiles of a run
  int32_t rows_by_tensor;       // wide kernel: contiguous activation rows come by tensor copies
  int32_t unit_cost;            // wide kernel: what a unit costs once, in row tiles
  int32_t resident;             // wide kernel: the weights of a unit's columns fit shared memory together
  int32_t vec_store;            // 16-byte stores of eight outputs are aligned
  int32_t quad_store;           // 8-byte stores of four outputs are aligned
  float* partial;               // fp32 sums of the column parts, or null: no column split
  size_t partial_bytes;
  const __half* col_scale;      // optional [rank]: activation rows are multiplied by it while staged
  int32_t rows_ready;           // decode kernel with column parts: route and activation rows were final then, only the stores wait
};

// Eight columns (8 * piece ..) of an activation row that cannot be copied as it is; `left`: how many of them exist.
// Permuted rows come in groups of 32 columns = 16 words of two halves 16 columns apart: a piece is the low or high
// halves of eight of them, read word by word.  Half by half a single projection of 64 experts x 256 rows took the
// tiled kernel 157 / 188 us (pair-interleaved / lane order), word by word 118 / 135; 16-byte loads were no faster (113 / 132) and ask
// for more alignment.
static __device__ __noinline__ uint4 read_piece(const TiledArgs& args, const __half* chunk, int c0, int piece, int left) {
  if (args.hidden_perm) {
    if (left <= 0) return make_uint4(0u, 0u, 0u, 0u);  // rank % 32 == 0: a group exists as a whole
    const uint32_t* grp = reinterpret_cast<const uint32_t*>(chunk + 32 * (piece >> 2));
    const uint32_t sel = (piece & 2) ? 0x7632u : 0x5410u;
    if (args.hidden_mode == TRIS_OUT_F16_PAIR_INTERLEAVED) {
      grp += 8 * (piece & 1);
      return make_uint4(prmt(grp[0], grp[1], sel), prmt(grp[2], grp[3], sel), prmt(grp[4], grp[5], sel), prmt(grp[6], grp[7], sel));
    }
    grp += (piece & 1) ? 0 : 1;
    return make_uint4(prmt(grp[0], grp[4], sel), prmt(grp[8], grp[12], sel), prmt(grp[2], grp[6], sel), prmt(grp[10], grp[14], sel));
  }
  uint32_t w[4] = {0u, 0u, 0u, 0u};
  for (int v = 0; v < 8 && v < left; ++v) {
    __half x = chunk[out_mode_pos(8 * piece + v, args.hidden_mode)];  // chunks start at multiples of 32 columns
    if (args.col_scale) x = __hmul(x, args.col_scale[c0 + 8 * piece + v]);
    w[v >> 1] |= static_cast<uint32_t>(__half_as_ushort(x)) << (16 * (v & 1));
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// ---- host helpers -----------------------------------------------------------------------------------
inline int sm_count() {
  static std::atomic<int> cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

template <typename Kernel>
int configure_smem(Kernel kernel, size_t smem, std::atomic<size_t> (&configured)[64]) {
  int dev = 0;
  TRIS_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || configured[dev].load(std::memory_order_relaxed) < smem) {
    TRIS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    if (dev >= 0 && dev < 64) configured[dev].store(smem, std::memory_order_relaxed);
  }
  return TRIS_OK;
}

constexpr size_t kMostSmem = 227 * 1024;

// Warps of a decode launch that splits neither columns nor passes.
inline long long decode_warps(const TiledArgs& args, int mode) {
  return static_cast<long long>((args.out_features + 31) / 32) * args.num_segments * (mode == MODE_SINGLE ? 1 : 2);
}
// A pass holds `rows` rows or more, 32 at most; args.row_split CTAs share the passes of a segment.  MODE_SINGLE,
// MODE_DUAL_STORE or MODE_DUAL_SILU.
int launch_grouped_decode(const TiledArgs& args, int mode, int rows, cudaStream_t stream, bool pdl);
constexpr int kDecodeMaxRows = 32;
// args.units_x, row_split, col_split, unit_cost and resident are set.
int launch_grouped_wide(const TiledArgs& args, int mode, int grid, cudaStream_t stream, bool pdl);
constexpr int kWideChunks = 2;  // chunks of 128 columns whose weights it can keep in shared memory

}  // namespace tr
}  // namespace tris
