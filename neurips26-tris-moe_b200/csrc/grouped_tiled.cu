// Grouped compact3 dequant-matmul over tile records, on the tcgen05 tensor cores, and the dump
// kernel the parity tests use.  See tile_records.cuh for the record layout and the unpack.
//
// Work unit = one expert segment x two output tiles of 128: the gate and the up tile of the same
// outputs (dual launch), or two neighbouring tiles of one projection.  A pass multiplies up to N rows
// of the segment; it walks the columns in chunks of 128, and a (pass, chunk) is an "item".  One
// persistent CTA per SM, its warps specialised so that the phases of consecutive items overlap:
//
//   loader (4 warps)     activation rows and column records of an item to shared memory (cp.async,
//                        a ring of stages), then the activations of the salient columns gathered
//                        into K columns of their own;
//   unpack (16 warps)    four warpgroups, one thread per output row: warpgroup (r, h) takes tile r of
//                        every second item.  A thread loads the code words of its own row straight from
//                        the record (coalesced, used once, so they never touch shared memory), unpacks
//                        64 columns to fp16 and writes them to its TMEM lane (tcgen05.st; two slots per
//                        warpgroup);
//   MMA (2 warps)        one per tile: tcgen05.mma with the weights from TMEM and the activations from shared memory
//                        into TMEM accumulators [128 outputs][rows];
//   epilogue (8 warps)   accumulators -> scale / bias or SiLU(gate) * up -> fp16 rows.
//
// No dequantised weight leaves the SM.  What bounds it: the roles' dependent steps, each on few warps, of which the unpack
// is the largest (3.9 lane-instructions per weight, against 16 for unpacking to mma.sync fragments with the
// Golomb-Rice decode in the loop).  509 tokens of 64 experts, gate/up and down: 28 / 27 us.
// Waits on mbarriers are bounded; a time-out is reported through the route's status word and the
// CTA leaves.
#include <math.h>

#include <type_traits>

#include "grouped_tiled.cuh"

namespace tris {
namespace tr {

constexpr int kUnpackWarps = 16, kLoadWarps = 4, kMmaWarps = 2;
// Warps of a CTA by role.  The narrow passes of decode need one epilogue warpgroup; with eight warps fewer
// than 32 every thread may use 72 registers, which is what the unpack wants.
template <int N>
struct Roles {
  static constexpr int kEpiWarps = N <= 64 ? 4 : 8;
  static constexpr int kEpi0 = kUnpackWarps, kLoad0 = kEpi0 + kEpiWarps, kMma0 = kLoad0 + kLoadWarps;
  static constexpr int kThreads = (kMma0 + kMmaWarps) * 32;
};
constexpr int kMaxStages = 4;
constexpr bool splits_columns(int n) { return n == 64; }  // whether an ordinary matrix with columns to split can come here
constexpr int kDBase = 4 * 2 * kACols;       // accumulators behind the four warpgroups' two slots
constexpr int kBarBytes = 512;               // barriers and the TMEM address
static_assert((2 * kMaxStages + 8 + 8 + 4 + 4 + kMmaWarps) * sizeof(uint64_t) + sizeof(uint32_t) <= kBarBytes, "barriers");
constexpr int kRowIdxBytes = 2 * 128 * 4;
constexpr int kOutBytes = 2 * 2 * 16 * kTileOut * 2;         // per epilogue warpgroup two tiles of 16 rows, fp16
constexpr int kHeadBytes = kBarBytes + kRowIdxBytes + kOutBytes + 1024;  // and the way to a 1024-byte boundary

// One stage: [activation rows: per 64 columns [N rows][128 B] in the 128-byte swizzle (piece p of row n at p ^ (n & 7))]
// [salient activations per projection: K-major core matrices, [column / 8][N rows][16 B]][column records].  In the
// swizzled form eight lanes fill one 128-byte line of shared memory from one line of global memory; as core
// matrices the two 16-byte halves of every sector went to different lines, and staging 128 rows x 128
// columns took 2600 cycles of 5200 an item has.
struct StageLayout {
  int col_bytes, col_off, rows_bytes, sal_off, sal_bytes, total;
};
__host__ __device__ inline StageLayout stage_layout(int max_steps, int ncol, int nset, int n) {
  StageLayout l;
  l.col_bytes = kColHdrBytes + kColTabBytes + max_steps * kColStepBytes;
  l.rows_bytes = n * kChunkCols * 2;
  l.sal_off = nset * l.rows_bytes;
  l.sal_bytes = max_steps * n * 32;
  l.col_off = l.sal_off + ncol * l.sal_bytes;
  l.total = (l.col_off + ncol * l.col_bytes + 1023) & ~1023;
  return l;
}

// Every role walks the same sequence: a CTA owns a contiguous range of units, and the units of one segment in
// it form a run; for every pass over the segment's rows, for every tile of the run, for every chunk: an item.
// The activation rows of a pass are staged once per run when all their chunks fit the ring (`reuse`),
// otherwise a run is one tile.  The route entries of the next run are loaded while the current one is
// worked on.
template <int N>
struct Walker {
  int u, u_end, nseg;
  int x, x_begin, x_end, expert, row_end, r0, c, c_begin, c_end, part;
  int next_x, next_expert, next_begin, next_end, next_part;
  __device__ __forceinline__ void peek(const TiledArgs& args, int unit) {
    if (unit >= u_end) return;
    const int q = unit / args.units_x;
    next_x = unit - q * args.units_x;
    int seg = q, z = 0;  // row split: part z takes the passes z, z + row_split, ...
    next_part = 0;       // column split: which part of the chunks
    if (args.row_split * args.col_split > 1) {
      z = q / nseg;
      seg = q - z * nseg;
      next_part = z / args.row_split;
      z -= next_part * args.row_split;
    }
    if (!args.expert_ids) {  // one segment of expert 0 with all rows
      next_expert = 0;
      next_begin = z * N;
      next_end = args.num_rows;
      return;
    }
    next_expert = args.expert_ids[seg];
    next_begin = args.segment_offsets[seg] + z * N;
    next_end = args.segment_offsets[seg + 1];
  }
  __device__ __forceinline__ void start(const TiledArgs& args) {
    nseg = args.num_segments_dev ? min(warp_uniform(*args.num_segments_dev), args.num_segments) : args.num_segments;
    const int total = nseg * args.units_x * args.row_split * args.col_split, per = total / gridDim.x, extra = total - per * gridDim.x;
    const int b = blockIdx.x;
    u = b * per + min(b, extra);
    u_end = u + per + (b < extra ? 1 : 0);
    peek(args, u);
    load(args);
  }
  __device__ __forceinline__ bool valid() const { return u < u_end; }
  __device__ __forceinline__ void load(const TiledArgs& args) {  // first item of the run at u, or of the next one that has rows
    while (u < u_end) {
      x = x_begin = next_x;  // (next_x comes from u; the loaded values are made uniform here, where they are first needed)
      x_end = args.reuse ? min(args.units_x, x_begin + (u_end - u)) : x_begin + 1;
      expert = warp_uniform(next_expert);
      r0 = warp_uniform(next_begin);
      row_end = min(warp_uniform(next_end), args.num_rows);
      part = next_part;
      c = c_begin = part * args.chunks / args.col_split;
      c_end = (part + 1) * args.chunks / args.col_split;
      peek(args, u + (x_end - x_begin));
      if (expert >= 0 && expert < args.num_experts && r0 < row_end) return;
      u += x_end - x_begin;
    }
  }
  __device__ __forceinline__ int rows() const { return min(N, row_end - r0); }
  __device__ __forceinline__ void next_pass(const TiledArgs& args) {
    c = c_begin;
    x = x_begin;
    r0 += args.row_split * N;
    if (r0 < row_end) return;
    u += x_end - x_begin;
    load(args);
  }
  __device__ __forceinline__ void next_tile(const TiledArgs& args) {
    c = c_begin;
    if (++x == x_end) next_pass(args);
  }
  __device__ __forceinline__ void next(const TiledArgs& args) {
    if (++c == c_end) next_tile(args);
  }
  __device__ __forceinline__ void next_stage(const TiledArgs& args) {  // for the role that does not look at tiles
    if (++c == c_end) next_pass(args);
  }
};

// Ring position: index and the parity of its current round.
struct Ring {
  int i = 0;
  uint32_t phase = 0u;
  __device__ __forceinline__ Ring at(int ahead, int n) const {  // ahead < n
    Ring r = *this;
    r.i += ahead;
    if (r.i >= n) {
      r.i -= n;
      r.phase ^= 1u;
    }
    return r;
  }
  __device__ __forceinline__ void advance(int n) {
    if (++i == n) {
      i = 0;
      phase ^= 1u;
    }
  }
};

// One chunk of a pass's activation rows; src[n] = source row of row n.  A warp covers 4 rows x 128
// contiguous bytes.  Rows that can be copied as they are (kVec) go by cp.async, anything else by read_piece;
// columns past the matrix read as zeros up to a multiple of 16.
template <int N, bool kVec>
__device__ __forceinline__ void stage_rows(const TiledArgs& args, uint8_t* dst, const __half* hidden, const int* src, int rows, int c0, int tid) {
  const int p = tid & 7, n0 = tid >> 3;
  const int cols = min(kChunkCols, args.rank - c0);
  dst += n0 * 128 + ((p ^ (n0 & 7)) << 4);
#pragma unroll 1
  for (int s = 0; s < 2; ++s, dst += N * 128) {
    const int piece = 8 * s + p, left = cols - 8 * piece;  // columns of this piece that exist
    if (left <= -8 || (left <= 0 && !(cols & 15))) return;
    uint8_t* d = dst;
    if constexpr (kVec) {
      // the row numbers of four copies first: one shared-memory round trip for all of them
      const __half* from = hidden + (left > 0 ? c0 + 8 * piece : 0);
#pragma unroll 1
      for (int n = n0; n < rows; n += 64, d += 64 * 128) {
        int r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) r[j] = src[min(n + 16 * j, N - 1)];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + 16 * j < rows) cp_async_16(d + 16 * 128 * j, from + static_cast<size_t>(r[j]) * args.hidden_stride, left > 0);
      }
    } else {
#pragma unroll 1
      for (int n = n0; n < rows; n += 16, d += 16 * 128)
        *reinterpret_cast<uint4*>(d) = read_piece(args, hidden + c0 + static_cast<size_t>(src[n]) * args.hidden_stride, c0, piece, left);
    }
  }
}

// Activations of the salient steps of one column record, [step * 2 + half][N rows][16 B].
template <int N>
__device__ __forceinline__ void gather_salient(uint8_t* dst, const uint8_t* rows_smem, const uint8_t* col, int rows, int tid) {
  const int items = reinterpret_cast<const ColHeader*>(col)->num_steps * 2 * N;
  for (int i = tid; i < items; i += kLoadWarps * 32) {
    const int n = i & (N - 1), kq = i / N;
    if (n >= rows) continue;
    const uint4 cols = *reinterpret_cast<const uint4*>(col + kColHdrBytes + kColTabBytes + (kq >> 1) * kColStepBytes + 64 + (kq & 1) * 16);
    const uint8_t* base = rows_smem + n * 128;
    auto ld = [&](uint32_t c) -> uint32_t {
      return *reinterpret_cast<const uint16_t*>(base + (c >> 6) * (N * 128) + ((((c >> 3) ^ n) & 7u) << 4) + (c & 7u) * 2);
    };
    auto pair = [&](uint32_t cc) { return ld(cc & 0xFFFFu) | (ld(cc >> 16) << 16); };
    *reinterpret_cast<uint4*>(dst + i * 16) = make_uint4(pair(cols.x), pair(cols.y), pair(cols.z), pair(cols.w));
  }
}

// N: activation rows per pass (the accumulators' TMEM columns).  A longer segment takes several
// passes and unpacks its weights again for each.  kVec: rows can be copied as they are; a variant of its own, because
// the call that reads other rows costs the kernel registers it does not have (spills; qkv 512 91 -> 94 us).
template <int N, int MODE, bool kVec>
__global__ void __launch_bounds__(Roles<N>::kThreads, 1) grouped_tiled_kernel(const __grid_constant__ TiledArgs args) {
  using W = Roles<N>;
  constexpr bool DUAL = MODE != MODE_SINGLE;
  constexpr int NC = DUAL ? 2 : 1;
  constexpr int kDBufs = (512 - kDBase) / (2 * N) < 4 ? (512 - kDBase) / (2 * N) : 4;
  extern __shared__ uint4 smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>(smem_raw);
  uint64_t* rows_full = reinterpret_cast<uint64_t*>(sm);   // loader -> MMA
  uint64_t* rows_empty = rows_full + kMaxStages;           // MMA (commits of both warps) -> loader
  uint64_t* a_full = rows_empty + kMaxStages;              // [warpgroup * 2 + slot] unpack warps -> MMA
  uint64_t* a_empty = a_full + 8;                          // MMA (commit) -> unpack
  uint64_t* d_full = a_empty + 8;                          // MMA (commit) -> epilogue
  uint64_t* d_empty = d_full + 4;                          // epilogue warps -> MMA
  uint64_t* mma_done = d_empty + 4;                        // [MMA warp] its last commit
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 2);
  int* src_rows = reinterpret_cast<int*>(sm + kBarBytes);  // [2][N] source rows of a pass, by pass parity
  uint8_t* stage_base = sm + ((smem_u32(sm) + kBarBytes + kRowIdxBytes + kOutBytes + 1023) & ~1023u) - smem_u32(sm);  // the swizzle counts from 1024-byte boundaries

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kMaxStages; ++i) {
      mbar_init(&rows_full[i], kLoadWarps);
      mbar_init(&rows_empty[i], 2);
    }
    for (int i = 0; i < 8; ++i) {
      mbar_init(&a_full[i], 4);
      mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&d_full[i], 2);
      mbar_init(&d_empty[i], W::kEpiWarps);
    }
    for (int i = 0; i < kMmaWarps; ++i) mbar_init(&mma_done[i], 1);
    fence_mbar_init();
  }
  if (warp == W::kMma0) tmem_alloc(tmem_slot, 512);  // before the dependents may start: they allocate too
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = warp_uniform(*tmem_slot);
  const StageLayout L = stage_layout(args.max_steps, NC, args.num_sets, N);
  bool ok = true;

  // The route and the activations come from earlier kernels.  When the route is older than the
  // predecessor, only the loader waits for it, so weights unpack while the predecessor still runs.
  if (!args.weights_before_wait) {
    pdl_wait();
    pdl_launch_dependents();
  }
  Walker<N> w;

  if (warp < kUnpackWarps) {
    // ---- unpack ---------------------------------------------------------------------------------
    const int wg = warp >> 2, r = wg & 1;
    const TrisProjView& v = args.proj[DUAL ? r : 0];
    const int max_sal = v.max_sal_words, rec_bytes = v.max_record_bytes, col_bytes = v.col_record_bytes;
    const int sal_off = record_slices(args.rank) * kSliceBytes, rows_off = sal_off + max_sal * kStepBytes;
    const uint32_t tmem_a = tmem + wg * (2 * kACols) + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    uint64_t* my_full = a_full + wg * 2;
    uint64_t* my_empty = a_empty + wg * 2;
    Ring slot;
    w.start(args);
    if (wg >> 1 && w.valid()) w.next(args);  // warpgroups 2 and 3 take the odd items
    // The column record is the same for all rows: broadcast loads through L1, where the other warps of the
    // SM find it too.  It and the first loads of the thread's own row are requested one item ahead.
    int nrec = -1, ncol = 0;  // record numbers
    uint32_t touched = 0u;    // one line of the next column record per lane: a load that only brings it to L1
    uint4 ncodes = make_uint4(0u, 0u, 0u, 0u);
    uint2 nscale = make_uint2(0u, 0u);
    // this warp's 32 output rows: sub-record warp % 4
    auto record = [&](int i) {
      return static_cast<const uint8_t*>(v.tile_records) + static_cast<size_t>(kSubs * i + (warp & 3)) * static_cast<size_t>(rec_bytes / kSubs);
    };
    auto column_record = [&](int i) { return static_cast<const uint8_t*>(v.col_records) + static_cast<size_t>(i) * static_cast<size_t>(col_bytes); };
    auto fetch = [&]() {
      const int tile = DUAL ? w.x : 2 * w.x + r;
      nrec = -1;
      if (!w.valid() || tile >= args.tiles) return;
      ncol = w.expert * args.chunks + w.c;
      nrec = (w.expert * args.tiles + tile) * args.chunks + w.c;
      const uint8_t* rec = record(nrec);
      if (lane * 128 < col_bytes) touched = __ldg(reinterpret_cast<const uint32_t*>(column_record(ncol) + lane * 128));
      ncodes = ldg_stream(rec + lane * 16);
      nscale = __ldg(reinterpret_cast<const uint2*>(rec + rows_off) + lane);
    };
    fetch();
    while (ok && w.valid()) {
      asm volatile("" ::"r"(touched));
      const int irec = nrec;
      const uint8_t* col = column_record(ncol);
      const int slices = (min(kChunkCols, args.rank - w.c * kChunkCols) + kSliceCols - 1) / kSliceCols;
      uint4 codes = ncodes, codes1 = ncodes;
      const uint2 rp0 = nscale;
      uint32_t sw0 = 0u, sw1 = 0u;
      if (irec >= 0) {
        const uint8_t* rec = record(irec);
        if (slices > 1) codes1 = ldg_stream(rec + kSliceBytes + lane * 16);
        if (max_sal > 0) sw0 = __ldg(reinterpret_cast<const uint32_t*>(rec + sal_off) + lane);
        if (max_sal > 1) sw1 = __ldg(reinterpret_cast<const uint32_t*>(rec + sal_off + kStepBytes) + lane);
      }
      w.next(args);
      if (w.valid()) w.next(args);
      fetch();
      if (irec < 0) continue;
      const uint4 hdr = __ldg(reinterpret_cast<const uint4*>(col));  // ColHeader: counts, slots of the packed rows, slots of the steps
      const uint32_t step_hi = __ldg(reinterpret_cast<const uint32_t*>(col) + 4);
      auto slot_scales = [&](uint32_t sl) {
        return sl == 0u ? rp0 : __ldg(reinterpret_cast<const uint2*>(record(irec) + rows_off + sl * kSlotBytes) + lane);
      };
      auto publish = [&]() {
        tmem_wait_st();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&my_full[slot.i]);
        slot.advance(2);
      };
      auto wait_slot = [&]() {
        ok = mbar_wait_warp(&my_empty[slot.i], slot.phase ^ 1u) && ok;
        tcgen05_fence_after();
      };
      const uint4* ct = reinterpret_cast<const uint4*>(col + kColHdrBytes);
      uint32_t row_slots = hdr.z;
#pragma unroll 1
      for (int s = 0; s < slices; ++s) {
        wait_slot();
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {  // rolled: the unpack of 32 columns is the loop body the instruction cache holds
          const RowScales rs = row_scales_ns(slot_scales(row_slots & 0xFFu));
          row_slots >>= 8;
          uint32_t a[16];
          unpack_word(codes.x, ct, rs, a);
          unpack_word(codes.y, ct + 1, rs, a + 8);
          tmem_st<16>(tmem_a + slot.i * kACols + h * 16, a);
          codes.x = codes.z;
          codes.y = codes.w;
          ct += 2;
        }
        ct += 12;
        codes = codes1;
        publish();
      }
      const int steps = static_cast<int>((hdr.y >> 8) & 0xFFu);
      uint32_t step_slots = hdr.w;
      const uint8_t* ent = col + kColHdrBytes + kColTabBytes;
#pragma unroll 1
      for (int b = 0; b < steps; b += 4) {
        wait_slot();
#pragma unroll 1
        for (int st = b; st < min(steps, b + 4); ++st) {
          const uint32_t code = st == 0 ? sw0 : (st == 1 ? sw1 : __ldg(reinterpret_cast<const uint32_t*>(record(irec) + sal_off + st * kStepBytes) + lane));
          uint32_t a[8];
          unpack_step(code, reinterpret_cast<const uint4*>(ent), slot_scales(step_slots & 0xFFu), a);
          tmem_st<8>(tmem_a + slot.i * kACols + (st - b) * 8, a);
          step_slots >>= 8;
          ent += kColStepBytes;
        }
        step_slots = step_hi;
        publish();
      }
    }
  } else if (warp < W::kLoad0) {
    // ---- epilogue -------------------------------------------------------------------------------
    // The buffer goes back as soon as its last accumulators are read: with rows of 128 there is one, and the
    // MMAs of the next tiles wait for it.  Results go through shared memory, from two rows of an output per word
    // to eight outputs of a row: 16-byte stores of whole lines.  With 4-byte stores after a shuffle, 8 rows at a
    // time, the epilogue of a unit took half the time between units (passes of 128 rows).
    const int e = (warp - W::kEpi0) >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t d_lane = tmem + kDBase + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    constexpr bool SILU = MODE == MODE_DUAL_SILU;
    constexpr int kParts = W::kEpiWarps / 4;  // warpgroups: each takes one projection or tile, or (SILU) every other 16 rows
    uint32_t* out_tile = reinterpret_cast<uint32_t*>(sm + kBarBytes + kRowIdxBytes) + e * (2 * 8 * kTileOut);
    int flip = 0;
    // 16 rows of a tile, as [pair of rows][output] words.  Two buffers: who writes one has passed the barrier
    // behind its last readers.
    auto store_tile = [&](__half* out, int tile, int r0, int n0, int rows, const float (&y)[16]) {
      uint32_t* b = out_tile + flip * (8 * kTileOut);
      flip ^= 1;
#pragma unroll
      for (int j = 0; j < 8; ++j) b[j * kTileOut + row] = h2_as_u32(__floats2half2_rn(y[2 * j], y[2 * j + 1]));
      named_barrier_sync(2 + e, 128);
      const int n = n0 + 2 * (row >> 4), o = tile * kTileOut + 8 * (row & 15);
      if (n >= rows || o >= args.out_features) return;
      const uint4* from = reinterpret_cast<const uint4*>(b + (row >> 4) * kTileOut + 8 * (row & 15));
      const uint4 p = from[0], q = from[1];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (n + k >= rows) break;
        const int to = args.out_scatter ? args.out_scatter[r0 + n + k] : r0 + n + k;
        if (to < 0) continue;
        const uint32_t sel = k ? 0x7632u : 0x5410u;
        const uint4 w8 = make_uint4(prmt(p.x, p.y, sel), prmt(p.z, p.w, sel), prmt(q.x, q.y, sel), prmt(q.z, q.w, sel));
        __half* dst = out + static_cast<size_t>(to) * args.out_features + o;
        if (args.vec_store) {
          *reinterpret_cast<uint4*>(dst) = w8;
        } else {
          const uint32_t h[4] = {w8.x, w8.y, w8.z, w8.w};
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (o + j < args.out_features) dst[j] = __ushort_as_half(static_cast<unsigned short>(h[j >> 1] >> (16 * (j & 1))));
        }
      }
    };
    Ring buf;
    for (w.start(args); w.valid(); w.next_tile(args)) {
      const int rows = w.rows(), expert = w.expert, x = w.x;
      const uint32_t d = d_lane + buf.i * (2 * N);
      ok = mbar_wait_warp<64>(&d_full[buf.i], buf.phase);
      if (named_barrier_or(2 + e, 128, !ok)) {  // the warps of a warpgroup leave together
        ok = false;
        break;
      }
      tcgen05_fence_after();
      const int per = (rows + 15) >> 4;  // steps of 16 rows
      const int halves = SILU ? 1 : (DUAL || 2 * x + 1 < args.tiles ? 2 : 1);
      const int steps = SILU ? (per + kParts - 1 - e) / kParts : (kParts == 1 ? halves * per : (e < halves ? per : 0));
      auto give_back = [&]() {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&d_empty[buf.i]);
      };
      // scale and bias of this thread's output, of either projection or tile
      float scale[2] = {1.f, 1.f}, bias[2] = {0.f, 0.f};
      bool scaled = false;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const TrisProjView& pv = args.proj[DUAL ? h : 0];
        if (args.partial || !(pv.output_scale || pv.bias)) continue;
        const int o = (DUAL ? x : 2 * x + h) * kTileOut + row;
        const size_t at = static_cast<size_t>(expert) * args.out_features + min(o, args.out_features - 1);
        if (pv.output_scale) scale[h] = __half2float(static_cast<const __half*>(pv.output_scale)[at]);
        if (pv.bias) bias[h] = __half2float(static_cast<const __half*>(pv.bias)[at]);
        scaled = true;
      }
      auto finish = [&](int h, float* y, int count) {
        if (!scaled) return;
#pragma unroll
        for (int j = 0; j < count; ++j) y[j] = y[j] * (h ? scale[1] : scale[0]) + (h ? bias[1] : bias[0]);
      };
#pragma unroll 1
      for (int i = 0; i < steps; ++i) {
        const int half = SILU ? 0 : (kParts == 1 ? i / per : e);
        const int n0 = 16 * (SILU ? e + kParts * i : (kParts == 1 ? i - half * per : i));
        float y[16];
        if constexpr (SILU) {
#pragma unroll
          for (int k = 0; k < 16; k += 8) {
            float g[8], up[8];
            tmem_ld_8_pair(d + n0 + k, d + N + n0 + k, g, up);
            finish(0, g, 8);
            finish(1, up, 8);
#pragma unroll
            for (int j = 0; j < 8; ++j) y[k + j] = __fdividef(g[j], 1.f + __expf(-g[j])) * up[j];
          }
        } else {
          tmem_ld_16(d + half * N + n0, y);
          finish(half, y, 16);
        }
        if (i + 1 == steps) give_back();
        if (splits_columns(N) && !SILU && args.partial) {  // a part of the columns: fp32 sums, [part][projection][row][output]
          const int o = (DUAL ? x : 2 * x + half) * kTileOut + row;
          float* dst = args.partial + (static_cast<size_t>(w.part * NC + (DUAL ? half : 0)) * args.num_rows + w.r0 + n0) * args.out_features + o;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (n0 + j < rows && o < args.out_features) dst[static_cast<size_t>(j) * args.out_features] = y[j];
          continue;
        }
        store_tile(args.out[DUAL ? half : 0], DUAL ? x : 2 * x + half, w.r0, n0, rows, y);
      }
      if (steps == 0) give_back();
      buf.advance(kDBufs);
    }
  } else if (warp < W::kMma0) {
    // ---- loader ---------------------------------------------------------------------------------
    const int tid = threadIdx.x - W::kLoad0 * 32;
    bool waited = !args.weights_before_wait;
    int next_src = 0, pass = 0;  // this thread's source row of the pass the walker has reached; that pass's parity
    auto find_row = [&]() {  // a plain load: a non-coherent one may be moved above the wait for the kernel that wrote the list
      if (w.valid() && tid < w.rows()) next_src = args.row_gather ? args.row_gather[w.r0 + tid] : w.r0 + tid;
    };
    auto keep_row = [&]() { if (tid < N) src_rows[pass * N + tid] = next_src; };
    uint32_t rows_of = 0u;  // rows of the items in flight, oldest in the low byte
    // Items requested before the oldest one in flight is handed over.  A stage of a reused pass is given back
    // only at the run's last tile, which needs all chunks of the pass handed over: the loader must not wait
    // for such a stage while it still holds one of the same pass back.
    const int ahead = min(args.stages - 1, args.reuse ? args.stages - args.pass_chunks + 1 : args.stages);
    Ring put, get;
    auto put_item = [&]() {
      if (w.valid()) {
        ok = mbar_wait_warp<32>(&rows_empty[put.i], put.phase ^ 1u) && ok;
        uint8_t* base = stage_base + put.i * L.total;
#pragma unroll 1
        for (int p = 0; p < NC; ++p) {
          const TrisProjView& pv = args.proj[p];
          const uint8_t* src = static_cast<const uint8_t*>(pv.col_records) + static_cast<size_t>(w.expert * args.chunks + w.c) * pv.col_record_bytes;
          for (int i = tid * 16; i < pv.col_record_bytes; i += kLoadWarps * 32 * 16) cp_async_16(base + L.col_off + p * L.col_bytes + i, src + i);
        }
        if (!waited) {
          pdl_wait();
          pdl_launch_dependents();
          waited = true;
        }
#pragma unroll 1
        for (int s = 0; s < args.num_sets; ++s)
          stage_rows<N, kVec>(args, base + s * L.rows_bytes, args.hidden[s], src_rows + pass * N, w.rows(), w.c * kChunkCols, tid);
        rows_of |= static_cast<uint32_t>(w.rows()) << (8 * ahead);
        w.next_stage(args);
        if (w.c == w.c_begin) {
          pass ^= 1;
          find_row();
        }
        put.advance(args.stages);
      }
      cp_async_commit();
      rows_of >>= 8;
    };
    w.start(args);
    if (args.weights_before_wait && args.row_gather) {  // the gather list may come from the predecessor
      pdl_wait();
      pdl_launch_dependents();
      waited = true;
    }
    find_row();
    for (int i = 0; i < ahead; ++i) {
      keep_row();
      named_barrier_sync(1, kLoadWarps * 32);
      put_item();
    }
    while (rows_of & 0xFFu) {
      keep_row();
      if (ahead == 1) cp_async_wait<0>();
      else if (ahead == 2) cp_async_wait<1>();
      else cp_async_wait<2>();
      // every loader thread's copies of this item have landed (and the loader warps leave together)
      if (named_barrier_or(1, kLoadWarps * 32, !ok)) {
        ok = false;
        break;
      }
      uint8_t* base = stage_base + get.i * L.total;
      const int rows = static_cast<int>(rows_of & 0xFFu);
#pragma unroll 1
      for (int p = 0; p < NC; ++p)
        gather_salient<N>(base + L.sal_off + p * L.sal_bytes, base + (args.num_sets == 2 ? p : 0) * L.rows_bytes,
                          base + L.col_off + p * L.col_bytes, rows, tid);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&rows_full[get.i]);
      get.advance(args.stages);
      put_item();
    }
    if (!waited) {
      pdl_wait();
      pdl_launch_dependents();
    }
    cp_async_wait<0>();
  } else {
    // ---- MMA ------------------------------------------------------------------------------------
    // A whole warp walks the items; one lane issues.  K steps of a full slice are unrolled: the operands of
    // an MMA live in uniform registers, and moving them there one by one costs more than the MMA.
    const int r = warp - W::kMma0;
    Ring stage, buf, slot0, slot1;
    uint32_t item = 0u;
    for (w.start(args); ok && w.valid(); ++item) {
      const int rows = w.rows(), cols = min(kChunkCols, args.rank - w.c * kChunkCols);
      const bool first = w.c == w.c_begin, last = w.c + 1 == w.c_end;
      const int pass_chunks = w.c_end - w.c_begin;
      const bool mine = DUAL || 2 * w.x + r < args.tiles, last_tile = w.x + 1 == w.x_end;
      const Ring at_stage = args.reuse ? stage.at(w.c - w.c_begin, args.stages) : stage;
      w.next(args);  // its route loads overlap the waits below
      const uint32_t idesc = umma_idesc_f16(kTileOut, (rows + 15) & ~15);
      const uint32_t d = tmem + kDBase + buf.i * (2 * N) + r * N;
      ok = mbar_wait_warp(&rows_full[at_stage.i], at_stage.phase);
      if (ok && first) ok = mbar_wait_warp(&d_empty[buf.i], buf.phase ^ 1u);
      if (!ok) break;
      const uint8_t* base = stage_base + at_stage.i * L.total;
      const int wg = static_cast<int>(item & 1u) * 2 + r;
      Ring sl = (item & 1u) ? slot1 : slot0;
      // one slot of weights: `n` K = 16 steps against the activations at desc, desc + step, ..
      auto consume = [&](int n, uint64_t desc, auto step, uint32_t accumulate) {
        constexpr int kStep = decltype(step)::value;
        const int at = wg * 2 + sl.i;
        ok = mbar_wait_warp(&a_full[at], sl.phase) && ok;
        tcgen05_fence_after();
        const uint32_t a = tmem + at * kACols;
        if (elect_one()) {
          umma_f16_ts(d, a, desc, idesc, accumulate);
          if (n == 4) {
#pragma unroll
            for (int j = 1; j < 4; ++j) umma_f16_ts(d, a + 8 * j, desc + j * kStep, idesc, 1u);
          } else {
            for (int j = 1; j < n; ++j) umma_f16_ts(d, a + 8 * j, desc + j * kStep, idesc, 1u);
          }
          umma_commit(&a_empty[at]);
        }
        sl.advance(2);
      };
      if (mine) {
        const uint32_t b_rows = smem_u32(base + (args.num_sets == 2 ? r : 0) * L.rows_bytes);
        for (int s = 0; s * kSliceCols < cols && ok; ++s)
          consume(min(kSliceCols / 16, (cols - s * kSliceCols + 15) >> 4), umma_smem_desc_sw128(b_rows + s * (N * 128)), std::integral_constant<int, 2>{},
                  first && s == 0 ? 0u : 1u);
        const int p = DUAL ? r : 0;
        const int steps = warp_uniform(reinterpret_cast<const ColHeader*>(base + L.col_off + p * L.col_bytes)->num_steps);
        const uint32_t b_sal = smem_u32(base + L.sal_off + p * L.sal_bytes);
        for (int b = 0; b < steps && ok; b += 4) consume(min(4, steps - b), umma_smem_desc(b_sal + b * (2 * N * 16), N * 16, 128), std::integral_constant<int, 2 * N>{}, 1u);
      }
      if (item & 1u) slot1 = sl;
      else slot0 = sl;
      if (elect_one()) {
        if (last_tile) umma_commit(&rows_empty[at_stage.i]);
        if (last) umma_commit(&d_full[buf.i]);
      }
      if (last) buf.advance(kDBufs);
      if (!args.reuse) stage.advance(args.stages);
      else if (last && last_tile) stage = stage.at(pass_chunks, args.stages);
    }
    // TMEM and shared memory go back below: not under an MMA that is still running, whichever role gave up
    if (elect_one()) umma_commit(&mma_done[r]);
    ok = mbar_wait_warp(&mma_done[r], 0u) && ok;
  }
  if (!ok && args.status) atomicExch(args.status, TRIS_ERR_TIMEOUT);
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  if (warp == W::kMma0) tmem_dealloc(tmem, 512);
}

// ---- dump kernel: dequantised weights from the records -----------------------------------------------
// grid (tiles, chunks, E), 128 threads; weights_out [E, O, rank]
__global__ void __launch_bounds__(kTileOut) tiled_dump_kernel(TrisProjView v, __half* weights_out) {
  extern __shared__ uint4 smem_raw[];
  uint8_t* col = reinterpret_cast<uint8_t*>(smem_raw);
  const int row = threadIdx.x, tile = blockIdx.x, c = blockIdx.y, e = blockIdx.z;
  const RecordGeom geo = record_geom(v);
  const uint8_t* rec = tile_record(v, geo, e, tile, c) + (row >> 5) * geo.sub_bytes;
  const uint8_t* src = col_record(v, geo, e, c);
  for (int i = row * 16; i < geo.col_bytes; i += kTileOut * 16) *reinterpret_cast<uint4*>(col + i) = *reinterpret_cast<const uint4*>(src + i);
  __syncthreads();
  const int o = tile * kTileOut + row;
  if (o >= v.out_features) return;
  const ColHeader* hdr = reinterpret_cast<const ColHeader*>(col);
  const int c0 = c * kChunkCols, cols = min(kChunkCols, v.rank - c0);
  __half* out = weights_out + (static_cast<size_t>(e) * v.out_features + o) * v.rank + c0;
  auto scales = [&](int slot) { return reinterpret_cast<const uint2*>(rec + geo.rows_off + slot * kSlotBytes)[row & 31]; };
  for (int w = 0; w < (cols + 15) / 16; ++w) {
    uint32_t a[8];
    unpack_word(reinterpret_cast<const uint32_t*>(rec + (w >> 2) * kSliceBytes + (row & 31) * 16)[w & 3],
                reinterpret_cast<const uint4*>(col + kColHdrBytes) + (w >> 2) * 16 + (w & 3), row_scales_ns(scales(hdr->slot_of_row[w >> 1])), a);
    for (int i = 0; i < 16; ++i)
      if (16 * w + i < cols) out[16 * w + i] = __ushort_as_half(static_cast<unsigned short>(a[i >> 1] >> (16 * (i & 1))));
  }
  for (int st = 0; st < hdr->num_steps; ++st) {  // the salient columns go over the +-0 the main unpack left there
    const uint8_t* ent = col + kColHdrBytes + kColTabBytes + st * kColStepBytes;
    uint32_t a[8];
    unpack_step(reinterpret_cast<const uint32_t*>(rec + geo.sal_off + st * kStepBytes)[row & 31], reinterpret_cast<const uint4*>(ent),
                scales(hdr->step_slot[st]), a);
    for (int i = 0; i < 16; ++i) {
      const unsigned at = reinterpret_cast<const uint16_t*>(ent + 64)[i];
      if (i > 0 && at == 0u) continue;  // unused position: columns ascend, so column 0 can only come first
      out[at] = __ushort_as_half(static_cast<unsigned short>(a[i >> 1] >> (16 * (i & 1))));
    }
  }
}

// ---- host side --------------------------------------------------------------------------------------
template <int MODE>
static size_t stage_bytes(const TiledArgs& args, int n) {
  return stage_layout(args.max_steps, MODE == MODE_SINGLE ? 1 : 2, args.num_sets, n).total;
}

// Row split: with fewer units than SMs - few local experts or one ordinary matrix, with long segments -
// up to g_row_split_max CTAs share a unit's row passes, each unpacking its weights for itself.
static std::atomic<int> g_row_split_max{4};
static int row_split(long long units, int max_rows, int n) {
  const int limit = g_row_split_max.load(std::memory_order_relaxed);
  if (limit <= 1 || units <= 0) return 1;
  return static_cast<int>(std::max<long long>(1, std::min<long long>({limit, sm_count() / units, (max_rows + n - 1) / n})));
}
// Rows of such a part on the weights-resident kernel.  Two row tiles would share an unpack where the columns do not fit shared
// memory, but half as many CTAs unpack then: 4096 x 4096, 256 rows 30.0 us with parts of 256, 25.1 with 128; a pair of 512 x 2048
// 22.6, 18.3; experts, 4096 x 320 x 2, a pair 17.7, 13.9.  (From 769 rows on there are four parts either way.)
constexpr int kPartRows = 128;

// Column split of one ordinary matrix (no experts): its units of two output tiles and its row passes together are
// too few for the SMs, and its columns many - parts of the columns go to CTAs of their own, whose fp32 sums
// sum_parts_kernel adds in order.  4096 columns, 512 rows: 64 CTAs for 4096 outputs (two parts), 32 for a pair of
// 1024 (four): 59 -> 39 and 61 -> 28 us.  At least two chunks per part: a part's sums are written and read once,
// 8 bytes per row and output (16 MB for 512 x 4096).
static size_t part_bytes(int num_rows, int out_features, int projections) { return sizeof(float) * static_cast<size_t>(projections) * num_rows * out_features; }
static long long col_parts(int chunks, long long units) { return std::min<long long>(chunks / 2, sm_count() / units); }
static int col_split(const TiledArgs& args, int mode, long long units) {
  if (args.expert_ids || !args.partial || units <= 0) return 1;
  const size_t part = part_bytes(args.num_rows, args.out_features, mode == MODE_SINGLE ? 1 : 2);
  return static_cast<int>(std::max<long long>(1, std::min<long long>(col_parts(args.chunks, units), static_cast<long long>(args.partial_bytes / part))));
}

// One thread per four outputs of a row: adds the parts, then scale, bias and SiLU * up as the epilogue would.
template <int MODE>
__global__ void __launch_bounds__(256) sum_parts_kernel(const __grid_constant__ TiledArgs args) {
  constexpr int P = MODE == MODE_SINGLE ? 1 : 2;
  const int quads = (args.out_features + 3) / 4;
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  const int row = static_cast<int>(i / quads), o = static_cast<int>(i - static_cast<long long>(row) * quads) * 4;
  pdl_wait();
  pdl_launch_dependents();
  if (row >= args.num_rows) return;
  const int to = args.out_scatter ? args.out_scatter[row] : row;
  if (to < 0) return;
  float y[P][4];
  const bool vec = args.out_features % 4 == 0;
#pragma unroll
  for (int p = 0; p < P; ++p) {
#pragma unroll
    for (int j = 0; j < 4; ++j) y[p][j] = 0.f;
    for (int k = 0; k < args.col_split; ++k) {
      const float* src = args.partial + (static_cast<size_t>(k * P + p) * args.num_rows + row) * args.out_features + o;
      if (vec) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(src));
        y[p][0] += v.x, y[p][1] += v.y, y[p][2] += v.z, y[p][3] += v.w;
      } else {
        for (int j = 0; j < 4 && o + j < args.out_features; ++j) y[p][j] += __ldcg(src + j);
      }
    }
    const TrisProjView& pv = args.proj[p];
    for (int j = 0; j < 4 && o + j < args.out_features; ++j) {
      if (pv.output_scale) y[p][j] *= __half2float(static_cast<const __half*>(pv.output_scale)[o + j]);
      if (pv.bias) y[p][j] += __half2float(static_cast<const __half*>(pv.bias)[o + j]);
    }
  }
  if constexpr (MODE == MODE_DUAL_SILU) {
#pragma unroll
    for (int j = 0; j < 4; ++j) y[0][j] = __fdividef(y[0][j], 1.f + __expf(-y[0][j])) * y[1][j];
  }
#pragma unroll
  for (int p = 0; p < (MODE == MODE_DUAL_STORE ? 2 : 1); ++p) {
    __half* dst = args.out[p] + static_cast<size_t>(to) * args.out_features + o;
    if (args.quad_store) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(h2_as_u32(__floats2half2_rn(y[p][0], y[p][1])), h2_as_u32(__floats2half2_rn(y[p][2], y[p][3])));
    } else {
      for (int j = 0; j < 4 && o + j < args.out_features; ++j) dst[j] = __float2half_rn(y[p][j]);
    }
  }
}

template <int N, int MODE, bool kVec>
static int launch_rows(const TiledArgs& args, int grid, size_t smem, cudaStream_t stream, bool pdl) {
  auto kernel = grouped_tiled_kernel<N, MODE, kVec>;
  static std::atomic<size_t> configured[64] = {};  // per instantiation, per device: largest size set so far
  const int st = configure_smem(kernel, smem, configured);
  if (st != TRIS_OK) return st;
  return check_cuda(launch_kernel(kernel, dim3(grid), dim3(Roles<N>::kThreads), smem, stream, pdl, 1, args), "grouped_tiled_kernel launch");
}
template <int N, int MODE>
static int launch_main(const TiledArgs& args, int grid, size_t smem, cudaStream_t stream, bool pdl) {
  return args.hidden_vec ? launch_rows<N, MODE, true>(args, grid, smem, stream, pdl) : launch_rows<N, MODE, false>(args, grid, smem, stream, pdl);
}

// Launches with the columns whole or split as args.col_split says: parts of gate and up are stored apart, the sum kernel
// applies SiLU * up.
template <int MODE, typename Launch>
static int launch_and_sum(TiledArgs& args, cudaStream_t stream, const Launch& launch) {
  if (args.col_split == 1) {
    args.partial = nullptr;
    return launch(std::integral_constant<int, MODE>{});
  }
  const int st = launch(std::integral_constant<int, MODE == MODE_DUAL_SILU ? MODE_DUAL_STORE : MODE>{});
  if (st != TRIS_OK) return st;
  const long long quads = static_cast<long long>(args.num_rows) * ceil_div(args.out_features, 4);
  return check_cuda(launch_kernel(sum_parts_kernel<MODE>, dim3(static_cast<unsigned>((quads + 255) / 256)), dim3(256), 0, stream, /*pdl=*/true, 1, args),
                    "sum_parts_kernel launch");
}

template <int N, int MODE>
static int launch_tiled(TiledArgs args, int max_rows, cudaStream_t stream, bool pdl) {
  const size_t stage = stage_bytes<MODE>(args, N);
  args.stages = static_cast<int>(std::min<size_t>(kMaxStages, (kMostSmem - kHeadBytes) / stage));
  TRIS_REQUIRE(args.stages >= 2, TRIS_ERR_UNSUPPORTED, "grouped_tiled_kernel: %zu bytes per stage", stage);
  const size_t smem = kHeadBytes + args.stages * stage;
  const long long units = static_cast<long long>(args.units_x) * args.num_segments;
  args.row_split = row_split(units, max_rows, N);
  // ordinary matrices of so many columns and more than 56 rows go to the weights-resident kernel
  args.col_split = splits_columns(N) ? col_split(args, MODE, units * args.row_split) : 1;
  args.pass_chunks = ceil_div(args.chunks, args.col_split);
  args.reuse = args.pass_chunks <= args.stages;
  const int grid = static_cast<int>(std::min<long long>(units * args.row_split * args.col_split, sm_count()));
  if constexpr (splits_columns(N)) {
    return launch_and_sum<MODE>(args, stream, [&](auto mode) { return launch_main<N, decltype(mode)::value>(args, grid, smem, stream, pdl); });
  } else {
    args.partial = nullptr;
    return launch_main<N, MODE>(args, grid, smem, stream, pdl);
  }
}

// Whether the weights-resident kernel is the faster one.  It pays about 5 us to start and its row tiles are 128 rows wide
// whatever a segment has; the tiled kernel unpacks a segment's weights again for every pass, of 64 rows where that is typical.
// So what counts is how many segments need one pass more than is typical, and whether the SMs have several units each to even that
// out: many experts.  us, tiled / wide, 64 experts, gate/up and down: 256 tokens (44 typical rows) 21.4 / 31.4, 21.6 / 26.3; 384
// (62: tails of 64-row passes) 35.3 / 32.2, 35.6 / 26.8; 509 (80) 28.2 / 32.4, 27.0 / 27.4; 700 (106) 46.1 / 36.7, 42.8 / 28.3;
// 2048 (288) 93.5 / 56.7, 90.0 / 43.0.  Whole blocks, tiled / wide: 64 experts, 57, 60 and 62 typical rows 95 / 87, 84 / 87, 100 /
// 88; 32 experts, 58, 62 and 70 53 / 64, 71 / 68, 65 / 70, at 110 and 120 66 / 70, 86 / 77; 8 experts, 106, 120 and 129 85 / 90, 94 /
// 97, 115 / 104.  One chunk of columns, 64 experts, gate/up and down: 400 and 1000 tokens 18.4 / 26.9, 17.6 / 20.4; 31.3 / 33.7, 34.1 /
// 24.6; blocks of 8 and 16 experts with down on either, 100 to 112 typical rows 67 / 67, 49 / 49 and 54 / 54, at 180 94 / 92, 58 / 56;
// with gate/up on either, at 180, 260 and 400 94 / 98, 110 / 113, 159 / 157 and 56 / 60, 69 / 74, 88 / 94.  Three chunks, 64 experts, 400
// tokens: 46.4 / 37.4, 31.2 / 31.0; 32 experts, 58, 70, 90 78 / 76, 72 / 72, 76 / 74; 16 experts, 80 54 / 54.
static bool wide_is_faster(const TiledArgs& args, int mode, int typical_rows) {
  const bool single = mode == MODE_SINGLE, many = args.num_segments >= 64;
  const int line = many ? 96 : (args.num_segments >= 32 ? 112 : 120);
  if (!args.expert_ids) {  // an ordinary matrix: 4096 columns, 100 rows 21.1 / 18.8, a pair 24.2 / 22.5
    if (args.chunks > kWideChunks) return typical_rows > 56;
    return typical_rows > (args.chunks == kWideChunks || single ? 96 : 160);
  }
  if (args.chunks == 1) return typical_rows > (single ? line : (many ? 160 : 400));
  // As many segments as SMs are uneven whatever their mean, but for gate/up the tiled kernel is the safer one as long as hardly any has a
  // second pass: 256 experts, blocks of 735 to 800 tokens (33 to 35) 143 to 210 us with tiled kernels, 143 to 173 with down on the wide
  // one, 154 to 158 with both (160 experts of 320 columns, 40: 124 / 128 / 140); from 820 (36) on the two are the same, 950 (41) 180 / 158 /
  // 158, 2048 (80) 273 / 211 / 196.
  if (args.num_segments >= sm_count()) return single || typical_rows > 40;
  if (typical_rows > (args.chunks > kWideChunks ? 96 : line)) return true;
  if (typical_rows <= 56) return false;
  return args.chunks > kWideChunks ? args.num_segments >= 32 : many && typical_rows <= 64;
}
template <int MODE>
static int launch_wide(TiledArgs args, int max_rows, cudaStream_t stream, bool pdl) {
  const long long units = static_cast<long long>(args.units_x) * args.num_segments;
  args.row_split = row_split(units, max_rows, kPartRows);
  args.col_split = col_split(args, MODE, units * args.row_split);
  args.resident = ceil_div(args.chunks, args.col_split) <= kWideChunks;
  args.unit_cost = MODE == MODE_SINGLE ? 2 : 1;  // unpacking a unit against a row tile, whose SiLU is the longer epilogue (44.7 / 34.4 us, 45.9 / 37.6 us the other way round: 1024 tokens)
  const int grid = static_cast<int>(std::min<long long>(units * args.row_split * args.col_split, sm_count()));
  return launch_and_sum<MODE>(args, stream, [&](auto mode) { return launch_grouped_wide(args, decltype(mode)::value, grid, stream, pdl); });
}

// Rows a decode pass should hold: a segment with more takes a second pass, and a launch as long as its longest segment, so it is the larger
// ones among all segments that count, the more of them the more; a wider pass makes the others slower.  Blocks in us, passes of 8 / 16 rows: 64
// experts, mean 3, 3.5 and 4 rows 38.5 / 41.1, 45.7 / 42.2, 47.3 / 43.4; 256 experts, 3 and 4 78.4 / 80.8, 86.9 / 82.9; 8 experts, 5 and 6 46.1 / 48.7,
// 51.7 / 49.3.  16 / 24 rows: 64 experts, 8 and 9 46.1 / 51.1, 54.9 / 51.8; 8 experts, 12 and 13 52.8 / 56.3, 60.4 / 56.8.  24 / 32 rows: 64
// experts, 15 and 16 59.2 / 57.7, 61.9 / 58.3 with one set of weights and 57.1 / 60.4 with another; 8 experts, 20 and 22 59.2 / 63.7, 69.1 / 66.2.
// Of other widths than two chunks of columns the wider pass costs more: 256 experts x 320 columns, 3.5 and 3.8 rows, 8 / 16 112.3 / 119.1,
// 109.4 / 116.0; 64 experts x 320, 3.5, 4 and 9 rows 57.0 / 60.9, 54.2 / 61.0, 70.5 / 73.0; 64 x 128, 9 rows, 16 / 24 39.4 / 41.6; 8 x 128,
// 20 rows, 24 / 32 56.4 / 54.7.
static int decode_rows(const TiledArgs& args, int max_rows) {
  const double mean = static_cast<double>(args.num_rows) / args.num_segments, sigma = sqrt(mean);
  const bool few = args.num_segments <= 16, many = args.num_segments >= 64 && args.chunks <= 2;
  const int plain = static_cast<int>(ceil(mean + 2.0 * sigma));
  int rows = few ? static_cast<int>(ceil(mean + (args.chunks == 1 ? 1.0 : 0.85) * sigma)) : many ? static_cast<int>(ceil(mean + 2.5 * sigma)) : plain;
  if (many && rows > 16) rows = args.chunks == 2 ? std::max(17, plain) : plain;
  return std::max(1, std::min(max_rows, rows));
}

template <int MODE>
static int dispatch_tiled(TiledArgs& args, int max_rows, int typical_rows, cudaStream_t stream, bool pdl) {
  args.units_x = MODE == MODE_SINGLE ? (args.tiles + 1) / 2 : args.tiles;
  args.row_split = 1;
  if (typical_rows <= kDecodeMaxRows) return launch_grouped_decode(args, MODE, decode_rows(args, max_rows), stream, pdl);
  // A few experts of up to 128 rows: passes of 32 rows, each in CTAs of its own, while all of them fit the SMs at once (20 warps
  // each with this tile, half of them the line because their columns are split too).  One expert with 128 rows, 4096 x 256:
  // 7.4 us against 12.1 on the tiled kernel, whose units are then fewer than the SMs.  At 14 warps the line would take
  // calls that the tiled kernel does in 11 us and this one in 13.
  const int passes = ceil_div(max_rows, kDecodeMaxRows);
  if (args.expert_ids && passes <= 4 && decode_warps(args, MODE) * passes <= 10ll * sm_count()) {
    args.row_split = passes;
    return launch_grouped_decode(args, MODE, kDecodeMaxRows, stream, pdl);
  }
  if (wide_is_faster(args, MODE, typical_rows)) return launch_wide<MODE>(args, max_rows, stream, pdl);
  // two stages of the widest pass have to fit shared memory (many salient columns make a stage larger)
  if (typical_rows <= 64 || 2 * stage_bytes<MODE>(args, 128) + kHeadBytes > kMostSmem) return launch_tiled<64, MODE>(args, max_rows, stream, pdl);
  return launch_tiled<128, MODE>(args, max_rows, stream, pdl);
}

}  // namespace tr

bool proj_has_tile_records(const TrisProjView& v) {
  return v.tile_records != nullptr && v.col_records != nullptr && v.use_block_gr && v.expert_slot == nullptr &&
         v.gmap_slot == nullptr && v.col_record_bytes > 0 && v.max_record_bytes > 0;
}

// mode: 0 single projection, 1 gate/up pair, 2 gate/up pair with SiLU * mul
int launch_grouped_tiled(const TrisProjView* proj_a, const TrisProjView* proj_b, const TrisRouteView* route,
                         const void* hidden_a, const void* hidden_b, void* out_a, void* out_b, int mode, int max_rows,
                         cudaStream_t stream, LaunchOpts opts) {
  using namespace tr;
  // Rows per pass: a longer segment costs a second pass that unpacks again, so size the pass for
  // mean + 2 sigma of a balanced router rather than for the worst case.
  int typical = max_rows;
  if (route->num_segments > 0) {
    const double mean = static_cast<double>(route->num_rows) / route->num_segments;
    typical = std::max(1, std::min(max_rows, static_cast<int>(ceil(mean + 2.0 * sqrt(mean)))));
  }
  TiledArgs a{};
  a.proj[0] = *proj_a;
  a.proj[1] = proj_b ? *proj_b : *proj_a;
  a.hidden[0] = static_cast<const __half*>(hidden_a);
  a.hidden[1] = static_cast<const __half*>(hidden_b ? hidden_b : hidden_a);
  a.out[0] = static_cast<__half*>(out_a);
  a.out[1] = static_cast<__half*>(out_b ? out_b : out_a);
  a.expert_ids = route->expert_ids;
  a.segment_offsets = route->segment_offsets;
  a.num_segments_dev = route->num_segments_dev;
  a.row_gather = route->row_gather;
  a.out_scatter = route->out_row_scatter;
  a.status = route->status_dev;
  a.num_segments = route->num_segments;
  a.num_rows = route->num_rows;
  a.rank = proj_a->rank;
  a.out_features = proj_a->out_features;
  a.num_experts = proj_a->num_experts;
  a.tiles = tiles_per_expert(a.out_features);
  a.chunks = num_chunks(a.rank);
  a.max_steps = std::max(a.proj[0].max_sal_words, a.proj[1].max_sal_words);
  a.max_sub_bytes = std::max(a.proj[0].max_record_bytes, a.proj[1].max_record_bytes) / kSubs;
  a.hidden_mode = (route->flags & TRIS_ROUTE_HIDDEN_LANE_ORDER)
                      ? TRIS_OUT_F16_LANE_ORDER
                      : ((route->flags & TRIS_ROUTE_HIDDEN_PAIR_INTERLEAVED) ? TRIS_OUT_F16_PAIR_INTERLEAVED : TRIS_OUT_F16);
  a.hidden_stride = route->hidden_row_stride > 0 ? route->hidden_row_stride : proj_a->rank;
  a.weights_before_wait = opts.pdl && opts.weights_before_wait;
  a.num_sets = (mode != MODE_SINGLE && a.hidden[0] != a.hidden[1]) ? 2 : 1;
  a.partial = static_cast<float*>(opts.workspace);
  a.partial_bytes = opts.workspace_bytes;
  a.col_scale = static_cast<const __half*>(route->hidden_col_scale);
  const uintptr_t rows_at = reinterpret_cast<uintptr_t>(a.hidden[0]) | reinterpret_cast<uintptr_t>(a.hidden[1]);
  a.hidden_vec = a.hidden_mode == TRIS_OUT_F16 && !a.col_scale && proj_a->rank % 8 == 0 && a.hidden_stride % 8 == 0 && (rows_at & 15u) == 0;
  a.hidden_perm = a.hidden_mode != TRIS_OUT_F16 && a.hidden_stride % 2 == 0 && (rows_at & 3u) == 0;
  a.rows_ready = a.weights_before_wait && opts.rows_ready;
  a.quad_store = proj_a->out_features % 4 == 0 && ((reinterpret_cast<uintptr_t>(a.out[0]) | reinterpret_cast<uintptr_t>(a.out[1])) & 7u) == 0;
  a.vec_store = proj_a->out_features % 8 == 0 && ((reinterpret_cast<uintptr_t>(a.out[0]) | reinterpret_cast<uintptr_t>(a.out[1])) & 15u) == 0;
  TRIS_REQUIRE(a.col_scale == nullptr || a.hidden_mode == TRIS_OUT_F16, TRIS_ERR_INVALID_ARG,
               "grouped (tile records): hidden_col_scale needs row-major activation rows");
  TRIS_REQUIRE(a.hidden_mode == TRIS_OUT_F16 || proj_a->rank % 32 == 0, TRIS_ERR_INVALID_ARG,
               "grouped (tile records): permuted activation rows need rank %% 32 == 0");
  TRIS_REQUIRE(a.hidden_stride >= proj_a->rank, TRIS_ERR_INVALID_ARG, "grouped (tile records): hidden_row_stride < rank");
  if (mode == MODE_SINGLE) return dispatch_tiled<MODE_SINGLE>(a, max_rows, typical, stream, opts.pdl);
  if (mode == MODE_DUAL_SILU) return dispatch_tiled<MODE_DUAL_SILU>(a, max_rows, typical, stream, opts.pdl);
  return dispatch_tiled<MODE_DUAL_STORE>(a, max_rows, typical, stream, opts.pdl);
}

int launch_tiled_dump(const TrisProjView* proj, void* weights_out, cudaStream_t stream) {
  using namespace tr;
  dim3 grid(tiles_per_expert(proj->out_features), num_chunks(proj->rank), proj->num_experts);
  tiled_dump_kernel<<<grid, kTileOut, proj->col_record_bytes, stream>>>(*proj, static_cast<__half*>(weights_out));
  return check_cuda(cudaGetLastError(), "tiled_dump_kernel launch");
}

}  // namespace tris

extern "C" int tris_set_grouped_row_split_max(int32_t ctas) {
  return tris::tr::g_row_split_max.exchange(ctas < 1 ? 1 : (ctas > 16 ? 16 : ctas), std::memory_order_relaxed);
}

// Bytes that let launch_grouped_tiled split the columns as far as it would: the parts of its launches (on the tiled kernel an
// ordinary matrix has too few rows for a second part, of 64 or of 128), within 256 MB.  The sums grow with the rows while
// the gain does not (100 000 rows of a 1024-output pair would ask for 3 GB); 4096 rows of a 4096 x 4096 matrix still get
// their two parts (134 MB).
constexpr size_t kMostSplitBytes = size_t{256} << 20;
size_t tris::grouped_split_bytes(const TrisProjView* proj, int projections, int num_rows) {
  using namespace tris::tr;
  if (!proj_has_tile_records(*proj) || num_rows <= kDecodeMaxRows || num_chunks(proj->rank) < 4) return 0;
  const long long tiles = tiles_per_expert(proj->out_features), units = projections == 1 ? (tiles + 1) / 2 : tiles;
  const size_t part = part_bytes(num_rows, proj->out_features, projections);
  const long long parts = std::min<long long>(col_parts(num_chunks(proj->rank), units * row_split(units, num_rows, kPartRows)),
                                              static_cast<long long>(kMostSplitBytes / part));
  return parts <= 1 ? 0 : part * static_cast<size_t>(parts);
}
