// Grouped compact3 dequant-matmul over tile records for segments of many rows, on the tcgen05 tensor cores:
// the dequantised weights of a unit stay in shared memory while all rows of its segment pass by.
//
// Work unit = one expert segment x two output tiles of 128: the gate and the up tile of the same outputs (dual
// launch), or two neighbouring tiles of one projection.  The activation rows are the M side of the MMA (128 rows = the
// TMEM lanes), the weights the N side.  One persistent CTA per SM, its warps specialised:
//
//   unpack (16 warps)    two groups of eight warps, each one 64-column slice of every chunk, a thread one output of one tile: code
//                        words from the record straight to fp16 in shared memory, in the 128-byte swizzle the MMA reads; the
//                        salient columns are then written over the +-0 the main unpack leaves there.  Four slots of a slice,
//                        that is two chunks;
//   tables (1 warp)      column scales and a list of the salient columns, per chunk, for the unpack;
//   loader (4 warps)     activation rows, 128 rows x 64 columns a stage, a ring of four: contiguous rows by tensor copies (one
//                        warp), gathered ones by cp.async;
//   MMA (1 warp)         tcgen05.mma, both operands from shared memory, accumulators [128 rows][2 x 128 outputs] in TMEM;
//   epilogue (8 warps)   accumulators -> scale / bias or SiLU(gate) * up -> fp16 rows.  A TMEM lane is a row, so eight
//                        outputs of a thread are 16 contiguous bytes.
//
// Up to 256 columns (the usual rank) the slots hold all of them: a unit is unpacked once however many rows its segment
// has, row tiles follow one another and two accumulator buffers let the epilogue of one run under the MMAs of the next.
// More columns stream through the slots; two row tiles at a time share a walk over the columns, each with an accumulator.
//
// No dequantised weight leaves the SM.  Waits on mbarriers are bounded; a time-out is reported through the route's
// status word and the CTA leaves.
//
// 2048 tokens of 64 experts, gate/up and down: 56.5 / 43.6 us, against 93.5 / 90.0 on the tiled kernel, which unpacks for every
// 128 rows and holds one accumulator buffer.  What bounds it: every role is a chain of dependent instructions, some 12
// cycles each between the other warps' (30 warps, issue slots 43 % busy, tensor pipe 20 / 29 %).  Taking work out, at a time when the two launches took 63.9 /
// 43.5: without the unpack 58 / 38, without the epilogue's work 46 / 32, without the products 57 / 38.  Without unpack and
// epilogue both 42 / 27: two thirds stay, the rows' way through loader, barriers and MMA warp, which every unit takes anew (gate/up
// of 2048 tokens: 160 row tiles x 8 units x 2 sets x 64 KB = 164 MB through two stages in flight per SM).  An SM is active for 77
// to 82 % of the longest one's time: units are shared out whole.
// Slower: shifting by multiplication on the other pipe (down 43.5 -> 47), listing the salient pairs
// twice to save the wrap-around (43.0 -> 46.9).
#include <cuda.h>

#include "grouped_tiled.cuh"

namespace tris {
namespace tr {
namespace wide {

constexpr int kUnpackWarps = 16, kEpiWarps = 8, kLoadWarps = 4;
constexpr int kEpi0 = kUnpackWarps, kLoad0 = kEpi0 + kEpiWarps, kMma0 = kLoad0 + kLoadWarps, kTable0 = kMma0 + 1;
constexpr int kThreads = (kTable0 + 1) * 32;
constexpr int kRows = 128;                          // rows of a row tile
constexpr int kBoxRows = 32;                        // of a tensor copy
constexpr int kLine = 2 * kSliceCols;               // 128 bytes: one row or output of a slice
constexpr int kTileBytes = kTileOut * kLine;        // one output tile of a slice
constexpr int kSlotBytes = 2 * kTileBytes;          // a slice of both tiles
constexpr int kSlots = 2 * kWideChunks;
constexpr int kStageBytes = kRows * kLine;
constexpr int kStages = 4;
constexpr int kEpiWarpBytes = 32 * 64;              // 32 rows x 64 bytes
// Of a chunk and projection: column scales as in the column record; for either slice a list of pairs of salient columns;
// {slots of the packed rows, pairs of slice 0 | steps << 16, pairs of slice 1, several slots?} and the slots of the steps.  A pair is
// {c1 scales, c2 scales, byte offsets of its columns in a line (kNoColumn: of the other slice, or none), place in its step |
// step << 8}.  A slice has at most 64 columns in two runs of equal group: 34 pairs and
// one that it shares.
constexpr int kPairBytes = 16, kListPairs = 36, kListBytes = kListPairs * kPairBytes;
constexpr int kPairsOff = kColTabBytes, kInfoOff = kPairsOff + 2 * kListBytes;
constexpr int kTableBytes = kInfoOff + 32;
constexpr uint32_t kNoColumn = 1u;                  // byte offsets of columns are even
constexpr int kStageOff = kSlots * kSlotBytes, kEpiOff = kStageOff + kStages * kStageBytes, kTableOff = kEpiOff + kEpiWarps * kEpiWarpBytes;
constexpr int kUnits = 4;                           // of the ring
constexpr int kUnitOff = kTableOff + 4 * kTableBytes, kBarOff = kUnitOff + kUnits * 32;
constexpr int kBarBytes = 512;
constexpr int kSmem = kBarOff + kBarBytes + 1024;   // and the way to a 1024-byte boundary
static_assert(kSmem <= 227 * 1024, "shared memory");
static_assert((2 * kStages + 2 * kSlots + 2 * kUnits + 9) * sizeof(uint64_t) + sizeof(uint32_t) <= kBarBytes, "barriers");
static_assert(kTableBytes % 16 == 0, "16-byte words");
constexpr int kGroupTiles = 2;                      // row tiles that share a walk over more columns than the slots hold

// A unit as the roles read it from the ring the planner fills.
struct Unit {
  int x, expert, r0, row_end;               // expert < 0: no more
  int c_begin, c_end, part, tiles;          // chunks; which part of them; row tiles
  __device__ __forceinline__ int tile_row(int step, int rt) const { return r0 + rt * step; }
  __device__ __forceinline__ int tile_rows(int step, int rt) const { return min(kRows, row_end - tile_row(step, rt)); }
};
static_assert(sizeof(Unit) == 32, "two 16-byte words");

struct Ring {  // index and the parity of its current round
  int i = 0;
  uint32_t phase = 0u;
  __device__ __forceinline__ void advance(int n) {
    if (++i == n) {
      i = 0;
      phase ^= 1u;
    }
  }
};

__device__ __forceinline__ bool mbar_test_at(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}
// Waits, bounded at about a second.  The hardware suspends the warp for up to the hinted time, so that a role that waits
// takes no issue slots from the roles it waits for.
__device__ __forceinline__ bool try_phase(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.b32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity), "r"(100000)
               : "memory");
  return ok != 0;
}
static __device__ __noinline__ bool wait_longer(uint32_t bar, uint32_t parity) {
  const uint32_t t0 = global_timer_lo();
  bool ok = false;
#pragma unroll 1
  do {
#pragma unroll 1
    for (int i = 0; i < 1024 && !ok; ++i) ok = try_phase(bar, parity);
  } while (!ok && global_timer_lo() - t0 < 1000000000u);
  return ok;
}
__device__ __forceinline__ bool wait_phase(uint64_t* bar, uint32_t parity) {
  const uint32_t at = smem_u32(bar);
  bool ok = try_phase(at, parity);
  if (!ok) ok = wait_longer(at, parity);
  return __all_sync(0xFFFFFFFFu, ok);
}
__device__ __forceinline__ void st_shared_v4(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void st_shared_u16_unless(uint32_t at, uint32_t v, uint32_t skip) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %2, 0;\n\t@p st.shared.b16 [%0], %1;\n\t}" ::"r"(at), "h"(static_cast<unsigned short>(v)), "r"(skip) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}

// Two floats in one register pair: one instruction for both.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// x / (1 + e^-x) * up for two outputs, with the hardware's 2^x and 1/x.  Where e^-x overflows its reciprocal is zero.
__device__ __forceinline__ void silu_mul(float& x0, float& x1, float up0, float up1) {
  const uint64_t x = pack2(x0, x1);
  float e0, e1, r0, r1;
  unpack2(mul2(x, pack2(-1.4426950408889634f, -1.4426950408889634f)), e0, e1);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e0));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e1));
  unpack2(add2(pack2(e0, e1), pack2(1.f, 1.f)), r0, r1);
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(r0));
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(r1));
  unpack2(mul2(mul2(x, pack2(r0, r1)), pack2(up0, up1)), x0, x1);
}

// The ring of units: every consumer warp takes each unit once.
struct Reader {
  uint32_t ring, full, empty, n = 0u;  // shared-memory addresses
  __device__ __forceinline__ Reader(uint32_t units, uint64_t* u_full, uint64_t* u_empty) : ring(units), full(smem_u32(u_full)), empty(smem_u32(u_empty)) {}
  __device__ __forceinline__ bool ready() const {
    return __all_sync(0xFFFFFFFFu, mbar_test_at(full + 8 * (n & (kUnits - 1)), (n / kUnits) & 1u));
  }
  __device__ __forceinline__ bool next(Unit& u) {
    const uint32_t at = n & (kUnits - 1), phase = (n / kUnits) & 1u;
    bool ok = try_phase(full + 8 * at, phase);
    if (!ok) ok = wait_longer(full + 8 * at, phase);
    const uint4 a = ld_shared_v4(ring + at * sizeof(Unit)), b = ld_shared_v4(ring + at * sizeof(Unit) + 16);
    __syncwarp();
    if (elect_one()) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + 8 * at) : "memory");
    ++n;
    u = {static_cast<int>(a.x), static_cast<int>(a.y), static_cast<int>(a.z), static_cast<int>(a.w),
         static_cast<int>(b.x), static_cast<int>(b.y), static_cast<int>(b.z), static_cast<int>(b.w)};
    if (!ok) u.expert = -2;  // the planner gave up
    return u.expert >= 0;
  }
};

// kVec: activation rows can be copied as they are.
template <int MODE, bool kVec>
__global__ void __launch_bounds__(kThreads, 1) grouped_wide_kernel(const __grid_constant__ TiledArgs args, const __grid_constant__ CUtensorMap rows_map) {
  constexpr bool DUAL = MODE != MODE_SINGLE;
  constexpr bool SILU = MODE == MODE_DUAL_SILU;
  constexpr int NC = DUAL ? 2 : 1;
  extern __shared__ uint4 smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>(smem_raw) + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // the swizzle counts from there
  uint64_t* a_full = reinterpret_cast<uint64_t*>(sm + kBarOff);  // loader -> MMA
  uint64_t* a_empty = a_full + kStages;                          // MMA (commit) -> loader
  uint64_t* w_full = a_empty + kStages;                          // unpack warps of a group -> MMA
  uint64_t* w_empty = w_full + kSlots;                           // MMA (commit) -> unpack
  uint64_t* t_full = w_empty + kSlots;                           // tables -> unpack
  uint64_t* t_empty = t_full + 2;                                // unpack warps -> tables
  uint64_t* d_full = t_empty + 2;                                // MMA (commit) -> epilogue
  uint64_t* d_empty = d_full + 2;                                // epilogue warps -> MMA
  uint64_t* u_full = d_empty + 2;                                // planner -> all
  uint64_t* u_empty = u_full + kUnits;                           // consumer warps -> planner
  uint64_t* mma_done = u_empty + kUnits;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    const int loaders = kVec && args.rows_by_tensor ? 1 : kLoadWarps;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&a_full[i], loaders);
      mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&w_full[i], kUnpackWarps / 2);
      mbar_init(&w_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&t_full[i], 1);
      mbar_init(&t_empty[i], kUnpackWarps);
      mbar_init(&d_full[i], 1);
      mbar_init(&d_empty[i], kEpiWarps);
    }
    for (int i = 0; i < kUnits; ++i) {
      mbar_init(&u_full[i], 1);
      mbar_init(&u_empty[i], kUnpackWarps + kEpiWarps + 1 + loaders);
    }
    mbar_init(mma_done, 1);
    fence_mbar_init();
  }
  if (warp == kMma0) tmem_alloc(tmem_slot, 512);  // before the dependents may start: they allocate too
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = warp_uniform(*tmem_slot);
  const uint32_t sm_at = warp_uniform(smem_u32(sm));
  bool ok = true;

  // The route and the activations come from earlier kernels.  When the route is older than the predecessor, only the
  // loader waits for it, so weights unpack while the predecessor still runs; nothing is stored before the loader's rows
  // have been multiplied.
  if (!args.weights_before_wait) {
    pdl_wait();
    pdl_launch_dependents();
  }
  const bool resident = args.resident;
  const int tile_step = kRows * args.row_split;  // rows from one row tile of a unit to the next
  Reader reader(sm_at + kUnitOff, u_full, u_empty);
  Unit w;

  if (warp < kUnpackWarps) {
    // ---- unpack ---------------------------------------------------------------------------------
    const int sl = warp >> 3, r = (warp >> 2) & 1;
    const TrisProjView& v = args.proj[DUAL ? r : 0];
    const int rec_bytes = v.max_record_bytes, max_sal = v.max_sal_words;
    const int sal_off = record_slices(args.rank) * tr::kSliceBytes, rows_off = sal_off + max_sal * kStepBytes;
    // this warp's 32 output rows: sub-record warp % 4
    const uint8_t* records = static_cast<const uint8_t*>(v.tile_records) + (warp & 3) * (rec_bytes / kSubs);
    const int row = (warp & 3) * 32 + lane;
    const uint32_t row_at = r * kTileBytes + row * kLine + ((row & 7) << 4);
    const uint32_t tables_at = sm_at + kTableOff + (DUAL ? r : 0) * kTableBytes, slots_at = sm_at + sl * kSlotBytes;
    // the thread's words of a chunk are asked for one chunk ahead
    w.c_begin = w.c_end = 0;
    const uint8_t* nrec = nullptr;  // null: no such tile or slice
    uint4 ncodes = make_uint4(0u, 0u, 0u, 0u);
    uint2 nscale = make_uint2(0u, 0u);
    uint32_t nsal = 0u;
    int c = 0, walks = 1;
    bool more = true;
    auto fetch = [&]() {
      nrec = nullptr;
      if (++c >= w.c_end) {
        c = w.c_begin;
        if (--walks == 0) {
          more = reader.next(w);
          c = w.c_begin;
          walks = resident ? 1 : (w.tiles + kGroupTiles - 1) / kGroupTiles;
        }
      }
      const int tile = DUAL ? w.x : 2 * w.x + r;
      if (!more || tile >= args.tiles || c * kChunkCols + sl * kSliceCols >= args.rank) return;
      nrec = records + static_cast<size_t>((w.expert * args.tiles + tile) * args.chunks + c) * static_cast<size_t>(rec_bytes);
      ncodes = ldg_stream(nrec + sl * tr::kSliceBytes + lane * 16);
      nscale = __ldg(reinterpret_cast<const uint2*>(nrec + rows_off) + lane);
      if (max_sal > 0) nsal = __ldg(reinterpret_cast<const uint32_t*>(nrec + sal_off) + lane);
    };
    fetch();
    uint32_t k = 0u;  // chunks so far
    while (ok && more) {
      const uint8_t* rec = nrec;
      uint4 codes = ncodes;
      const uint2 rp0 = nscale;
      const uint32_t sal0 = nsal;
      fetch();
      const uint32_t pair = k & 1u, phase = (k >> 1) & 1u;
      ok = wait_phase(&t_full[pair], phase);
      ok = wait_phase(&w_empty[2 * pair + sl], phase ^ 1u) && ok;
      if (rec != nullptr) {
        const uint32_t table_at = tables_at + pair * (2 * kTableBytes), at = slots_at + pair * (2 * kSlotBytes) + row_at;  // bases are multiples of 1024: byte b of the line at ^ b
        const uint4 info = ld_shared_v4(table_at + kInfoOff);
        const bool several = info.w != 0u;
        auto slot_scales = [&](uint32_t s) {
          return s == 0u ? rp0 : __ldg(reinterpret_cast<const uint2*>(rec + rows_off + s * tr::kSlotBytes) + lane);
        };
        RowScales rs = row_scales_ns(rp0);
        uint32_t row_slots = info.x >> (16 * sl), ct = table_at + sl * (kColTabBytes / 2);
#pragma unroll 1
        for (int h = 0; h < 128; h += 64) {  // rolled: the unpack of 32 columns is the loop body the instruction cache holds
          if (several) rs = row_scales_ns(slot_scales(row_slots & 0xFFu));
          row_slots >>= 8;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            uint32_t a[8];
            const uint32_t w = i ? codes.y : codes.x;
#pragma unroll
            for (int j = 0; j < 4; ++j) unpack_two(w << (2 * j), w << (2 * j + 1), ld_shared_v4(ct + i * 16 + j * 64), rs, a[2 * j], a[2 * j + 1]);
            st_shared_v4(at ^ (h + i * 32), a[0], a[1], a[2], a[3]);
            st_shared_v4(at ^ (h + i * 32 + 16), a[4], a[5], a[6], a[7]);
          }
          codes.x = codes.z;
          codes.y = codes.w;
          ct += 32;
        }
        // Salient columns.  A column of 32 rows lies in 8 banks; the quarters of a warp, 8 rows each, start at different
        // pairs so that their stores fall into different banks most of the time.
        const uint32_t pairs = (sl ? info.z : info.y) & 0xFFFFu, steps = info.y >> 16;
        if (pairs != 0u) {
          const uint32_t begin = table_at + kPairsOff + sl * kListBytes, end = begin + pairs * kPairBytes;
          uint32_t ent = begin + (((lane >> 3) * pairs) >> 2) * kPairBytes;
          auto patch = [&](const uint4& e, uint32_t code, __half2 r1, __half2 r2) {
            const uint32_t t = __funnelshift_l(0u, code, e.w);  // by the low bits: the place
            const uint32_t p1 = flip_by_sign(h2_as_u32(__hmul2_rn(u32_as_h2(e.x), r1)), t);
            const uint32_t p2 = flip_by_sign(h2_as_u32(__hmul2_rn(u32_as_h2(e.y), r2)), t << 8);
            const uint32_t y = h2_as_u32(__hadd2_rn(u32_as_h2(p1), u32_as_h2(p2)));
            st_shared_u16_unless(at ^ (e.z & 0xFFFFu), y, e.z & kNoColumn);
            st_shared_u16_unless(at ^ (e.z >> 16), y >> 16, e.z & (kNoColumn << 16));
          };
          auto r1_of = [&](uint2 rp) { return u32_as_h2(prmt(rp.x, 0u, 0x1010u)); };
          auto r2_of = [&](uint2 rp) { return u32_as_h2(prmt(rp.x, 0u, 0x3232u)); };
          auto code_of = [&](uint32_t st) { return __ldg(reinterpret_cast<const uint32_t*>(rec + sal_off + st * kStepBytes) + lane); };
          auto following = [&](uint32_t e) { return e + kPairBytes == end ? begin : e + kPairBytes; };
          if (!several && steps <= 2u) {  // the next pair is on its way while one is written
            const uint32_t sal1 = steps == 2u ? code_of(1u) : 0u;
            const __half2 r1 = r1_of(rp0), r2 = r2_of(rp0);
            uint4 e = ld_shared_v4(ent);
#pragma unroll 1
            for (uint32_t i = pairs;;) {
              ent = following(ent);
              const uint4 f = ld_shared_v4(ent);
              patch(e, e.w >= 256u ? sal1 : sal0, r1, r2);
              if (--i == 0u) break;
              ent = following(ent);
              e = ld_shared_v4(ent);
              patch(f, f.w >= 256u ? sal1 : sal0, r1, r2);
              if (--i == 0u) break;
            }
          } else {
#pragma unroll 1
            for (uint32_t i = 0; i < pairs; ++i, ent = following(ent)) {
              const uint4 e = ld_shared_v4(ent), step_slots = ld_shared_v4(table_at + kInfoOff + 16);
              const uint32_t st = e.w >> 8;
              const uint2 rp = slot_scales(((st < 4u ? step_slots.x : step_slots.y) >> (8u * (st & 3u))) & 0xFFu);
              patch(e, code_of(st), r1_of(rp), r2_of(rp));
            }
          }
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&w_full[2 * pair + sl]);
        mbar_arrive(&t_empty[pair]);
      }
      ++k;
    }
  } else if (warp == kTable0) {
    // ---- planner and tables ---------------------------------------------------------------------
    // Units in order of segment, then of output: neighbours share their rows and column records.  A CTA gets the units that
    // start within its share of the cost, an equal part of the sum over all: segments differ in their rows.  With rows or
    // columns split there is one unit per CTA.
    uint32_t k = 0u, produced = 0u;
    auto publish = [&](const Unit& u) {
      const uint32_t at = produced & (kUnits - 1);
      ok = wait_phase(&u_empty[at], ((produced / kUnits) & 1u) ^ 1u) && ok;
      if (lane == 0) {
        st_shared_v4(sm_at + kUnitOff + at * sizeof(Unit), u.x, u.expert, u.r0, u.row_end);
        st_shared_v4(sm_at + kUnitOff + at * sizeof(Unit) + 16, u.c_begin, u.c_end, u.part, u.tiles);
        mbar_arrive(&u_full[at]);
      }
      ++produced;
    };
    int built[2] = {-1, -1};  // record a buffer was made from: units of a segment share their tables
    auto build = [&](int record) {
      const uint32_t b = k & 1u;
      ok = wait_phase(&t_empty[b], ((k >> 1) & 1u) ^ 1u);
      if ((b ? built[1] : built[0]) != record) {
#pragma unroll 1
        for (int p = 0; p < NC; ++p) {
          const TrisProjView& v = args.proj[p];
          const uint8_t* col = static_cast<const uint8_t*>(v.col_records) + static_cast<size_t>(record) * static_cast<size_t>(v.col_record_bytes);
          const uint4 hdr = __ldg(reinterpret_cast<const uint4*>(col));  // ColHeader: counts, slots of the packed rows, slots of the steps
          const uint32_t more_slots = __ldg(reinterpret_cast<const uint32_t*>(col) + 4);
          const uint4 tab = __ldg(reinterpret_cast<const uint4*>(col + kColHdrBytes) + lane);
          uint2 scales[2];
          uint32_t cols[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int st = 4 * i + (lane >> 3), j = lane & 7;
            const uint8_t* ent = col + kColHdrBytes + kColTabBytes + st * kColStepBytes;
            const bool in = st < v.max_sal_words;
            scales[i] = in ? __ldg(reinterpret_cast<const uint2*>(ent) + j) : make_uint2(0u, 0u);
            cols[i] = in ? __ldg(reinterpret_cast<const uint32_t*>(ent + 64) + j) : 0u;
          }
          const uint32_t to = sm_at + kTableOff + (2 * b + p) * kTableBytes;
          st_shared_v4(to + lane * 16, tab.x, tab.y, tab.z, tab.w);
          const int steps = static_cast<int>((hdr.y >> 8) & 0xFFu);
          uint32_t count[2] = {0u, 0u};
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            // Columns ascend over the steps of a chunk; places that stay empty name column 0, which can only come first.
            const int st = 4 * i + (lane >> 3), j = lane & 7;
            const uint32_t c0 = cols[i] & 0xFFFFu, c1 = cols[i] >> 16;
            const bool in0 = st < steps && (c0 != 0u || j == 0), in1 = st < steps && c1 != 0u;
#pragma unroll
            for (uint32_t s = 0; s < 2; ++s) {
              const bool mine0 = in0 && (c0 >> 6) == s, mine1 = in1 && (c1 >> 6) == s;
              const uint32_t who = __ballot_sync(0xFFFFFFFFu, mine0 || mine1), at = count[s] + __popc(who & ((1u << lane) - 1u));
              if ((mine0 || mine1) && at < kListPairs)
                st_shared_v4(to + kPairsOff + s * kListBytes + at * kPairBytes, scales[i].x, scales[i].y,
                             (mine0 ? 2u * (c0 & 63u) : kNoColumn) | ((mine1 ? 2u * (c1 & 63u) : kNoColumn) << 16), j | (st << 8));
              count[s] += __popc(who);
            }
          }
          if (lane == 0) {
            st_shared_v4(to + kInfoOff, hdr.z, min(count[0], kListPairs) | (static_cast<uint32_t>(steps) << 16), min(count[1], kListPairs), (hdr.y & 0xFFu) > 1u ? 1u : 0u);
            st_shared_v4(to + kInfoOff + 16, hdr.w, more_slots, 0u, 0u);
          }
        }
        (b ? built[1] : built[0]) = record;
        __syncwarp();
      }
      if (lane == 0) mbar_arrive(&t_full[b]);
      ++k;
    };
    const int nseg = args.num_segments_dev ? min(warp_uniform(*args.num_segments_dev), args.num_segments) : args.num_segments;
    const bool arrays = args.expert_ids != nullptr, split = args.row_split * args.col_split > 1;  // no arrays: one segment of expert 0 with all rows
    auto expert_of = [&](int seg) { return seg >= nseg ? -1 : (arrays ? args.expert_ids[seg] : 0); };
    auto begin_of = [&](int seg) { return seg >= nseg || !arrays ? 0 : args.segment_offsets[seg]; };
    auto end_of = [&](int seg) { return seg >= nseg ? 0 : (arrays ? min(args.segment_offsets[seg + 1], args.num_rows) : args.num_rows); };
    auto cost_of = [&](int rows) { return rows > 0 ? args.unit_cost + (rows + kRows - 1) / kRows : 0; };
    int z = 0, part = 0, lo = 0, hi = 0, at = 0, s0 = 0;  // at: cost of the units before segment s0
    if (split) {  // the unit that this CTA has, with a cost of 1 for each
      const int q = blockIdx.x / args.units_x, y = q / nseg;
      part = y / args.row_split;
      z = y - part * args.row_split;
      s0 = q - y * nseg;
      lo = blockIdx.x - q * args.units_x;
      hi = part < args.col_split ? lo + 1 : 0;
    } else {
      int sum = 0;
      for (int s = lane; s < nseg; s += 32) sum += cost_of(end_of(s) - begin_of(s));
      sum = __reduce_add_sync(0xFFFFFFFFu, sum) * args.units_x;
      lo = static_cast<int>(static_cast<long long>(sum) * blockIdx.x / gridDim.x);
      hi = static_cast<int>(static_cast<long long>(sum) * (blockIdx.x + 1) / gridDim.x);
    }
    const int c_begin = part * args.chunks / args.col_split, c_end = (part + 1) * args.chunks / args.col_split;
#pragma unroll 1
    for (; s0 < nseg && at < hi && ok; s0 += 32) {
      const int expert = expert_of(s0 + lane), begin = begin_of(s0 + lane), finish = end_of(s0 + lane);
      const int cost = split ? (lane == 0) : cost_of(finish - begin), group = __reduce_add_sync(0xFFFFFFFFu, cost) * args.units_x;
#pragma unroll 1
      for (int i = 0, a = at; i < 32 && a < hi && at + group > lo && ok; ++i) {
        const int per = __shfl_sync(0xFFFFFFFFu, cost, i);
        Unit u{0, __shfl_sync(0xFFFFFFFFu, expert, i), __shfl_sync(0xFFFFFFFFu, begin, i) + z * kRows, __shfl_sync(0xFFFFFFFFu, finish, i), c_begin, c_end, part, 0};
        u.tiles = (u.row_end - u.r0 + tile_step - 1) / tile_step;
        if (per > 0 && a + per * args.units_x > lo && u.r0 < u.row_end && u.expert >= 0 && u.expert < args.num_experts) {
          const int walks = resident ? 1 : (u.tiles + kGroupTiles - 1) / kGroupTiles;
#pragma unroll 1
          for (u.x = a >= lo ? 0 : (lo - a + per - 1) / per; u.x < args.units_x && a + u.x * per < hi && ok; ++u.x) {
            publish(u);
#pragma unroll 1
            for (int y = 0; y < walks && ok; ++y)
#pragma unroll 1
              for (int c = c_begin; c < c_end && ok; ++c) build(u.expert * args.chunks + c);
          }
        }
        a += per * args.units_x;
      }
      at += group;
    }
    publish(Unit{0, -1, 0, 0, 0, 0, 0, 0});
  } else if (warp < kLoad0) {
    // ---- epilogue -------------------------------------------------------------------------------
    // Warp (q, h): rows 32 q .. + 31 of the row tile and, of the outputs, tile h or (SiLU) half h of the tile.  32 outputs
    // of 32 rows at a time go through 2 KB of the warp's own, so that a row is stored as 64 contiguous bytes: 16-byte
    // stores of 32 different rows would take the L1 32 cycles each.
    const int q = warp & 3, h = (warp - kEpi0) >> 2;
    const uint32_t d_lane = tmem + (static_cast<uint32_t>(q * 32) << 16);
    uint8_t* buf_w = sm + kEpiOff + (warp - kEpi0) * kEpiWarpBytes;
    const uint32_t put_at = smem_u32(buf_w) + lane * 64;                      // piece p of row n at p ^ ((n >> 1) & 3)
    const uint32_t put_x = ((lane >> 1) & 3) << 4;
    const int get_row = lane >> 2, get_piece = lane & 3;
    const uint8_t* get_at = buf_w + get_row * 64 + ((get_piece ^ ((get_row >> 1) & 3)) << 4);  // rows get_row + 8 i: the same swizzle
    Ring buf;
    while (ok && reader.next(w)) {
      const int tiles = w.tiles, x = w.x;
      const int tile = DUAL ? x : 2 * x + h;
      const bool present = DUAL || tile < args.tiles;
#pragma unroll 1
      for (int rt = 0; rt < tiles; ++rt) {
        const int row0 = w.tile_row(tile_step, rt) + q * 32, live = min(32, w.tile_rows(tile_step, rt) - q * 32);
        ok = wait_phase(&d_full[buf.i], buf.phase);
        if (!ok) break;
        tcgen05_fence_after();
        const uint32_t d = d_lane + buf.i * 256;
        auto give_back = [&]() {
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&d_empty[buf.i]);
        };
        if (live <= 0 || !present) {
          give_back();
          buf.advance(2);
          continue;
        }
        // scale and bias of the outputs from o0 on, of projection or tile `half`
        auto finish = [&](int half, int o0, float* y, int count) {
          const TrisProjView& pv = args.proj[DUAL ? half : 0];
          if (!(pv.output_scale || pv.bias)) return;
          for (int j = 0; j < count; ++j) {
            const size_t at = static_cast<size_t>(w.expert) * args.out_features + min(o0 + j, args.out_features - 1);
            if (pv.output_scale) y[j] *= __half2float(__ldg(static_cast<const __half*>(pv.output_scale) + at));
            if (pv.bias) y[j] += __half2float(__ldg(static_cast<const __half*>(pv.bias) + at));
          }
        };
        if (!SILU && args.partial) {  // a part of the columns: fp32 sums, [part][projection][row][output]
          float* dst = args.partial + (static_cast<size_t>(w.part * (DUAL ? 2 : 1) + (DUAL ? h : 0)) * args.num_rows + row0) * args.out_features;
#pragma unroll 1
          for (int b = 0; b < kTileOut; b += 16) {
            float y[16];
            tmem_ld_16(d + h * kTileOut + b, y);
            if (b + 16 == kTileOut) give_back();
#pragma unroll
            for (int p = 0; p < 4; ++p)
              st_shared_v4(put_at + ((p << 4) ^ put_x), __float_as_uint(y[4 * p]), __float_as_uint(y[4 * p + 1]), __float_as_uint(y[4 * p + 2]), __float_as_uint(y[4 * p + 3]));
            __syncwarp();
            const int o = tile * kTileOut + b + 4 * get_piece;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int n = get_row + 8 * i;
              if (n < live && o < args.out_features) {
                const float4 s = *reinterpret_cast<const float4*>(get_at + i * 8 * 64);
                float* to = dst + static_cast<size_t>(n) * args.out_features + o;
                if (args.out_features % 4 == 0) {
                  *reinterpret_cast<float4*>(to) = s;
                } else {
                  const float f[4] = {s.x, s.y, s.z, s.w};
                  for (int j = 0; j < 4 && o + j < args.out_features; ++j) to[j] = f[j];
                }
              }
            }
            __syncwarp();
          }
          buf.advance(2);
          continue;
        }
        constexpr int kOuts = SILU ? kTileOut / 2 : kTileOut;  // of this warp
        const int first = SILU ? h * kOuts : 0;                // within the tile
        const int o_first = tile * kTileOut + first;
        __half* to[4];  // this lane's four rows, its piece of the first 32 outputs; null: no such row
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int n = get_row + 8 * i, row = n >= live ? -1 : (args.out_scatter ? args.out_scatter[row0 + n] : row0 + n);
          to[i] = row < 0 ? nullptr : args.out[MODE == MODE_DUAL_STORE ? h : 0] + static_cast<size_t>(row) * args.out_features + o_first + 8 * get_piece;
        }
        const uint32_t d_at = d + (SILU ? first : h * kTileOut);
#pragma unroll 1
        for (int b = 0; b < kOuts; b += 16) {
          float y[16], up[SILU ? 16 : 1];
          if constexpr (SILU) tmem_ld_16_pair(d_at + b, d_at + kTileOut + b, y, up);
          else tmem_ld_16(d_at + b, y);
          if (b + 16 == kOuts) give_back();
          uint32_t z[8];
          if constexpr (SILU) {
            finish(0, o_first + b, y, 16);
            finish(1, o_first + b, up, 16);
#pragma unroll
            for (int j = 0; j < 16; j += 2) silu_mul(y[j], y[j + 1], up[j], up[j + 1]);
          } else {
            finish(DUAL ? h : 0, o_first + b, y, 16);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) z[j] = h2_as_u32(__floats2half2_rn(y[2 * j], y[2 * j + 1]));
          const uint32_t half = (b & 16) << 1;  // of the 64-byte lines
          st_shared_v4(put_at + (half ^ put_x), z[0], z[1], z[2], z[3]);
          st_shared_v4(put_at + ((half + 16) ^ put_x), z[4], z[5], z[6], z[7]);
          if (half == 0u) continue;
          __syncwarp();
          const int o = o_first + (b - 16) + 8 * get_piece;
          if (o < args.out_features) {
            uint4 s[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i] = *reinterpret_cast<const uint4*>(get_at + i * 8 * 64);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (to[i] == nullptr) continue;
              __half* dst = to[i] + (b - 16);
              if (args.vec_store) {
                *reinterpret_cast<uint4*>(dst) = s[i];
              } else {
                const uint32_t u[4] = {s[i].x, s[i].y, s[i].z, s[i].w};
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  if (o + j < args.out_features) dst[j] = __ushort_as_half(static_cast<unsigned short>(u[j >> 1] >> (16 * (j & 1))));
              }
            }
          }
          __syncwarp();
        }
        buf.advance(2);
      }
    }
  } else if (warp < kMma0) {
    // ---- loader ---------------------------------------------------------------------------------
    // A stage is 128 rows x 64 columns of one set.  Contiguous rows: one warp asks for boxes of 32 rows.  Otherwise a
    // warp copies every fourth group of four rows, 128 contiguous bytes of each at a time; copies of up to two stages
    // are in flight behind the one asked for, and a warp that finds the ring full first hands over what it has, so that it
    // never waits for a stage that waits for it.
    Ring put;
    bool waited = !args.weights_before_wait;
    if (!waited) {  // rows and gather list come from the predecessor
      pdl_wait();
      pdl_launch_dependents();
    }
    const int group = resident ? 1 : kGroupTiles;
    if (kVec && args.rows_by_tensor) {
      while (warp == kLoad0 && ok && reader.next(w)) {
        const int tiles = w.tiles, slice_end = min(2 * w.c_end, (args.rank + kSliceCols - 1) / kSliceCols);
#pragma unroll 1
        for (int t0 = 0; t0 < tiles && ok; t0 += group)
#pragma unroll 1
          for (int s = 2 * w.c_begin; s < slice_end && ok; ++s)
#pragma unroll 1
            for (int rt = t0; rt < min(tiles, t0 + group) && ok; ++rt) {
              ok = wait_phase(&a_empty[put.i], put.phase ^ 1u);
              const int boxes = (w.tile_rows(tile_step, rt) + kBoxRows - 1) / kBoxRows;
              if (ok && lane == 0) mbar_arrive_expect_tx(&a_full[put.i], boxes * kBoxRows * kLine);
              __syncwarp();
              if (ok && lane < boxes)
                tma_load_2d(sm + kStageOff + put.i * kStageBytes + lane * kBoxRows * kLine, &rows_map, s * kSliceCols, w.tile_row(tile_step, rt) + lane * kBoxRows, &a_full[put.i]);
              put.advance(kStages);
            }
      }
      // shared memory goes back below: not under a copy that is still on its way
      for (int i = 0; i < kStages && warp == kLoad0; ++i) wait_phase(&a_full[i], i < put.i ? put.phase : put.phase ^ 1u);
    } else {
      const int piece = lane & 7, n0 = (warp - kLoad0) * 4 + (lane >> 3);
      const uint32_t put_at = sm_at + kStageOff + n0 * kLine + ((piece ^ (n0 & 7)) << 4);  // rows n0 + 16 i: the same swizzle
      constexpr int kInFlight = kStages - 2;
      Ring get;
      int pending = 0;
      auto hand_over = [&]() {
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[get.i]);
        get.advance(kStages);
        --pending;
      };
      auto hand_over_all = [&]() {
        cp_async_wait<0>();
        while (pending > 0) hand_over();
      };
      auto next_unit = [&]() {  // the planner may be waiting for products of the rows still held
        if (!reader.ready()) hand_over_all();
        return reader.next(w);
      };
      while (ok && next_unit()) {
        const int tiles = w.tiles, slice_begin = 2 * w.c_begin, slice_end = min(2 * w.c_end, (args.rank + kSliceCols - 1) / kSliceCols);
#pragma unroll 1
        for (int t0 = 0; t0 < tiles && ok; t0 += group) {
          const __half* src[8] = {};
          int rows = 0;
#pragma unroll 1
          for (int s = slice_begin; s < slice_end && ok; ++s)
#pragma unroll 1
            for (int rt = t0; rt < min(tiles, t0 + group) && ok; ++rt) {
              const int row0 = w.tile_row(tile_step, rt);
              if (kVec && (!resident || s == slice_begin)) {
                rows = w.tile_rows(tile_step, rt);
#pragma unroll
                for (int i = 0; i < 8; ++i) {  // plain loads: non-coherent ones may be moved above the wait for the kernel that wrote the list
                  const int n = min(n0 + 16 * i, rows - 1);
                  src[i] = args.hidden[0] + static_cast<size_t>(args.row_gather ? args.row_gather[row0 + n] : row0 + n) * args.hidden_stride;
                }
              }
#pragma unroll 1
              for (int set = 0; set < args.num_sets && ok; ++set) {
                uint64_t* empty = &a_empty[put.i];
                if (!__all_sync(0xFFFFFFFFu, mbar_test_at(smem_u32(empty), put.phase ^ 1u))) {
                  hand_over_all();
                  ok = wait_phase(empty, put.phase ^ 1u) && ok;
                }
                const int c0 = s * kSliceCols, at = c0 + 8 * piece, left = args.rank - at;  // columns of this piece that exist
                if (8 * piece < ((min(kSliceCols, args.rank - c0) + 15) & ~15)) {           // read as zeros up to a multiple of 16
                  const uint32_t dst = put_at + put.i * kStageBytes;
                  if constexpr (kVec) {
                    const ptrdiff_t off = (left > 0 ? at : 0) + (set ? args.hidden[1] - args.hidden[0] : 0);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                      if (n0 + 16 * i < rows)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + i * 16 * kLine), "l"(src[i] + off), "r"(left > 0 ? 16 : 0) : "memory");
                  } else {
                    const int chunk0 = c0 & ~(kChunkCols - 1), here = w.tile_rows(tile_step, rt);
#pragma unroll 1
                    for (int n = n0, i = 0; n < here; n += 16, ++i) {
                      const int from = args.row_gather ? args.row_gather[row0 + n] : row0 + n;
                      const uint4 y = read_piece(args, args.hidden[set] + chunk0 + static_cast<size_t>(from) * args.hidden_stride, chunk0, (at - chunk0) >> 3, left);
                      st_shared_v4(dst + i * 16 * kLine, y.x, y.y, y.z, y.w);
                    }
                  }
                }
                cp_async_commit();
                put.advance(kStages);
                if (++pending > kInFlight) {
                  cp_async_wait<kInFlight>();
                  hand_over();
                }
              }
            }
        }
      }
      hand_over_all();
    }
  } else {
    // ---- MMA ------------------------------------------------------------------------------------
    // A whole warp walks the stages; one lane issues.  With one set of rows the two tiles of outputs are one N = 256
    // operand.  The control of a stage is on the way of every row tile: an instruction takes some 12 cycles between the
    // other roles' warps.
    uint32_t k = 0u, n = 0u, turn = 0u;  // chunks, stages and row tiles so far
    const bool two_sets = args.num_sets == 2, leader = elect_one();
    const uint64_t stages_desc = umma_smem_desc_sw128(sm_at + kStageOff), slots_desc = umma_smem_desc_sw128(sm_at);
    const uint32_t bars = smem_u32(a_full);
    auto wait_at = [&](uint32_t bar, uint32_t parity) {
      bool there = try_phase(bar, parity);
      if (!__all_sync(0xFFFFFFFFu, there)) ok = __all_sync(0xFFFFFFFFu, there || wait_longer(bar, parity)) && ok;
    };
    auto at_of = [&](const uint64_t* first, uint32_t i) { return bars + static_cast<uint32_t>(reinterpret_cast<const uint8_t*>(first) - reinterpret_cast<const uint8_t*>(a_full)) + 8 * i; };
    // one stage: a slice of a row tile against one tile of outputs (two sets of rows) or both
    auto multiply = [&](uint32_t d, uint64_t db, uint32_t idesc, int steps, uint32_t accumulate) {
      const uint32_t at = n & (kStages - 1);
      wait_at(at_of(a_full, at), (n / kStages) & 1u);
      tcgen05_fence_after();
      const uint64_t da = stages_desc + at * (kStageBytes >> 4);
      if (leader) {
        umma_f16_ss(d, da, db, idesc, accumulate);
        if (steps == 4) {
#pragma unroll
          for (int j = 1; j < 4; ++j) umma_f16_ss(d, da + 2 * j, db + 2 * j, idesc, 1u);
        } else {
          for (int j = 1; j < steps; ++j) umma_f16_ss(d, da + 2 * j, db + 2 * j, idesc, 1u);
        }
        umma_commit(&a_empty[at]);
      }
      ++n;
    };
    while (ok && reader.next(w)) {
      const int tiles = warp_uniform(w.tiles), c_begin = warp_uniform(w.c_begin), slices = 2 * (warp_uniform(w.c_end) - c_begin);
      const uint32_t idesc = umma_idesc_f16(kRows, two_sets || !(DUAL || 2 * warp_uniform(w.x) + 1 < args.tiles) ? kTileOut : 2 * kTileOut);
      const int left = args.rank - c_begin * kChunkCols, live = min(slices, (left + kSliceCols - 1) / kSliceCols);  // slices that exist
      auto slot_of = [&](int i) { return 2 * ((k + (i >> 1)) & 1u) + (i & 1u); };
      auto wait_weights = [&](int i) { wait_at(at_of(w_full, slot_of(i)), ((k + (i >> 1)) >> 1) & 1u); };
      auto free_weights = [&](int i) {
        if (leader) umma_commit(&w_empty[slot_of(i)]);
      };
      auto wait_accumulator = [&](uint32_t t) { wait_at(at_of(d_empty, t & 1u), ((t >> 1) & 1u) ^ 1u); };
      if (resident) {  // the slots are the slices in order, behind each other
        const int shift = two_sets ? 1 : 0, items = live << shift;
        const uint64_t db0 = slots_desc + slot_of(0) * (kSlotBytes >> 4);
        const uint64_t db_step = (two_sets ? kTileBytes : kSlotBytes) >> 4;
#pragma unroll 1
        for (int rt = 0; rt < tiles && ok; ++rt, ++turn) {
          wait_accumulator(turn);
          const uint32_t d = tmem + (turn & 1u) * 256;
          const bool fresh = rt == 0, done = rt + 1 == tiles;  // weights: first and last use
          uint64_t db = db0;
#pragma unroll 1
          for (int i = 0; i < items && ok; ++i, db += db_step) {
            const int s = i >> shift, second = i & shift;
            if (fresh && !second) wait_weights(s);
            multiply(d + second * kTileOut, db, idesc, min(4, (left - s * kSliceCols + 15) >> 4), s > 0 ? 1u : 0u);
            if (done && second == shift) free_weights(s);
          }
          if (ok && leader) umma_commit(&d_full[turn & 1u]);
        }
        for (int i = live; i < slices && ok; ++i) {
          wait_weights(i);
          free_weights(i);
        }
        k += slices >> 1;
      } else {
#pragma unroll 1
        for (int t0 = 0; t0 < tiles && ok; t0 += kGroupTiles, k += slices >> 1) {
          const int here = min(kGroupTiles, tiles - t0);
#pragma unroll 1
          for (int i = 0; i < slices && ok; ++i) {
            wait_weights(i);
            const uint64_t db = slots_desc + slot_of(i) * (kSlotBytes >> 4);
            const int steps = min(4, (left - i * kSliceCols + 15) >> 4);
#pragma unroll 1
            for (int rt = 0; rt < here && i < live && ok; ++rt) {
              if (i == 0) wait_accumulator(turn + rt);
              const uint32_t d = tmem + ((turn + rt) & 1u) * 256;
              multiply(d, db, idesc, steps, i > 0 ? 1u : 0u);
              if (two_sets) multiply(d + kTileOut, db + (kTileBytes >> 4), idesc, steps, i > 0 ? 1u : 0u);
            }
            free_weights(i);
          }
          for (int rt = 0; rt < here; ++rt, ++turn)
            if (ok && leader) umma_commit(&d_full[turn & 1u]);
        }
      }
    }
    // TMEM and shared memory go back below: not under an MMA that is still running, whichever role gave up
    if (leader) umma_commit(mma_done);
    ok = wait_phase(mma_done, 0u) && ok;
  }
  if (!ok && args.status) atomicExch(args.status, TRIS_ERR_TIMEOUT);
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  if (warp == kMma0) tmem_dealloc(tmem, 512);
}

template <int MODE>
static int launch(TiledArgs args, int grid, cudaStream_t stream, bool pdl) {
  CUtensorMap rows_map{};
  args.rows_by_tensor = args.hidden_vec && args.row_gather == nullptr && args.num_sets == 1 &&
                        encode_rows_map(&rows_map, args.hidden[0], args.num_rows, args.rank, args.hidden_stride, kBoxRows);
  auto kernel = args.hidden_vec ? grouped_wide_kernel<MODE, true> : grouped_wide_kernel<MODE, false>;
  static std::atomic<size_t> configured[2][64] = {};
  const int st = configure_smem(kernel, kSmem, configured[args.hidden_vec ? 1 : 0]);
  if (st != TRIS_OK) return st;
  return check_cuda(launch_kernel(kernel, dim3(grid), dim3(kThreads), kSmem, stream, pdl, 1, args, rows_map), "grouped_wide_kernel launch");
}
}  // namespace wide

int launch_grouped_wide(const TiledArgs& args, int mode, int grid, cudaStream_t stream, bool pdl) {
  if (mode == MODE_SINGLE) return wide::launch<MODE_SINGLE>(args, grid, stream, pdl);
  if (mode == MODE_DUAL_SILU) return wide::launch<MODE_DUAL_SILU>(args, grid, stream, pdl);
  return wide::launch<MODE_DUAL_STORE>(args, grid, stream, pdl);
}

}  // namespace tr
}  // namespace tris
