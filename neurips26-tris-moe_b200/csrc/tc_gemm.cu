// Backbone projection on the 5th-generation tensor cores (tcgen05 + TMEM), used when there
// are enough activation rows for a dense contraction (prefill, or the down backbone over
// all routed rows of a decode batch): out[n, m] = sum_k x[n, k] * A[m, k].
//
// One CTA computes a 128-output x NTILE-row tile over its share of K.  Operands are staged
// in shared memory in the K-major no-swizzle ("interleaved") core-matrix layout: 8 rows x
// 16 bytes per core matrix, all rows of one 8-column K chunk contiguous, so
//   byte offset(row, k) = (k / 8) * ROWS * 16 + row * 16 + (k % 8) * 2,
// stride between 8-row groups (SBO) = 128 B, stride between K chunks (LBO) = ROWS * 16 B.
// A single thread issues tcgen05.mma (M = 128, N = NTILE, K = 16 per instruction) into a
// TMEM accumulator; completion is tracked with tcgen05.commit on mbarriers, two shared-memory
// stages deep, so the loads of chunk i+1 overlap the MMAs of chunk i.  The split-K partial
// tiles of a thread-block cluster are reduced through distributed shared memory.
// Every mbarrier wait is bounded; a time-out frees the TMEM allocation and reports
// TRIS_ERR_TIMEOUT through the status word.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "umma.cuh"

namespace cg = cooperative_groups;

namespace tris {

struct TcGemmArgs {
  SkinnyProblem prob[3];
  int32_t num_problems;
  const __half* x;
  const int32_t* row_gather;
  const int32_t* n_dev;
  int32_t* status;
  int32_t n;
  int32_t k;
  int32_t k_per_cta;  // multiple of kTcKChunk
  int32_t a_before_wait;  // the matrices are older than the predecessor kernel
};

constexpr int kTcStages = 4;

template <int NTILE>
struct alignas(128) TcSmem {
  uint8_t a[kTcStages][kTcM * kTcKChunk * 2];
  uint8_t b[kTcStages][NTILE * kTcKChunk * 2];
  uint64_t mbar[kTcStages];
  uint32_t tmem_base;
  int32_t timed_out;
};

// Accumulator -> fp32 partial tile in shared memory -> (cluster reduction over the K split) ->
// outputs.  `part` is the CTA's shared memory from its start (the stage buffers are free by now).
template <int NTILE>
__device__ __forceinline__ void tc_gemm_epilogue(const TcGemmArgs& args, const SkinnyProblem& pb, float* part,
                                                 uint32_t tmem, bool failed, int nchunks, int m0, int n0, int n_live,
                                                 cg::cluster_group& cluster) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // accumulator -> fp32 partial tile in shared memory, [NTILE][128] (stage buffers are free now)
  if (!failed && nchunks > 0) {
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
#pragma unroll 1
    for (int c0 = 0; c0 < NTILE; c0 += 16) {
      float v[16];
      tmem_ld_16(tmem + lane_base + c0, v);
#pragma unroll
      for (int j = 0; j < 16; ++j) part[(c0 + j) * kTcM + warp * 32 + lane] = v[j];
    }
  } else {
    for (int i = threadIdx.x; i < NTILE * kTcM; i += kTcThreads) part[i] = 0.f;
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, NTILE);
  if (failed && threadIdx.x == 0 && args.status) atomicExch(args.status, TRIS_ERR_TIMEOUT);

  cluster.sync();
  {
    // every CTA of the cluster reduces and stores its own slice of the tile; the remote
    // reads of one element are independent, so they are all in flight together
    const unsigned nblk = cluster.num_blocks(), rank = cluster.block_rank();
    constexpr int kVec = NTILE * kTcM / 4;
    const int per = (kVec + nblk - 1) / nblk;
    const int v_end = min(kVec, static_cast<int>((rank + 1) * per));
    const float4* parts[8];
#pragma unroll
    for (unsigned r = 0; r < 8; ++r)
      parts[r] = reinterpret_cast<const float4*>(cluster.map_shared_rank(part, r < nblk ? r : 0));
    for (int i4 = rank * per + threadIdx.x; i4 < v_end; i4 += kTcThreads) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      if (NTILE == 128 && nblk == 1) {  // the columns are not split: no eight predicated remote reads of which one counts (64 rows: 10.0 us without the branch, 10.2 with it)
        acc = reinterpret_cast<const float4*>(part)[i4];
      } else {
        float4 v[8];
#pragma unroll
        for (unsigned r = 0; r < 8; ++r) v[r] = (r < nblk) ? parts[r][i4] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (unsigned r = 0; r < 8; ++r) { acc.x += v[r].x; acc.y += v[r].y; acc.z += v[r].z; acc.w += v[r].w; }
      }
      const int n = n0 + (4 * i4) / kTcM, mbase = m0 + (4 * i4) % kTcM;
      if (n >= n_live) continue;
      if ((pb.m & 3) == 0 && mbase < pb.m && (pb.out_mode == TRIS_OUT_F32 || pb.out_mode == TRIS_OUT_F16)) {
        const size_t at = static_cast<size_t>(n) * pb.m + mbase;
        if (pb.out_mode == TRIS_OUT_F32) {
          if ((reinterpret_cast<uintptr_t>(pb.out) & 15u) == 0) {
            *reinterpret_cast<float4*>(static_cast<float*>(pb.out) + at) = acc;
            continue;
          }
        } else if ((reinterpret_cast<uintptr_t>(pb.out) & 7u) == 0) {
          *reinterpret_cast<uint2*>(static_cast<__half*>(pb.out) + at) =
              make_uint2(h2_as_u32(__floats2half2_rn(acc.x, acc.y)), h2_as_u32(__floats2half2_rn(acc.z, acc.w)));
          continue;
        }
      }
      const float vals[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int m = mbase + u;
        if (m >= pb.m) continue;
        if (pb.out_mode == TRIS_OUT_F32) {
          static_cast<float*>(pb.out)[static_cast<size_t>(n) * pb.m + m] = vals[u];
        } else {
          const int mm = out_mode_pos(m, pb.out_mode);
          static_cast<__half*>(pb.out)[static_cast<size_t>(n) * pb.m + mm] = __float2half_rn(vals[u]);
        }
      }
    }
  }
  cluster.sync();  // keep every CTA's shared memory alive until its peers have read it
}

// grid (m tiles over all problems, ceil(n / NTILE), ksplit); cluster (1, 1, ksplit).
// After the MMAs the stage buffers are reused as the fp32 partial tile [NTILE][128].
template <int NTILE>
__global__ void __launch_bounds__(kTcThreads) umma_gemm_kernel(const __grid_constant__ TcGemmArgs args) {
  extern __shared__ uint4 smem_raw[];
  auto& sm = *reinterpret_cast<TcSmem<NTILE>*>(smem_raw);
  cg::cluster_group cluster = cg::this_cluster();
  const int warp = threadIdx.x >> 5;

  int tile = blockIdx.x, pi = 0;
  while (pi + 1 < args.num_problems && tile >= (args.prob[pi].m + kTcM - 1) / kTcM) {
    tile -= (args.prob[pi].m + kTcM - 1) / kTcM;
    ++pi;
  }
  const SkinnyProblem& pb = args.prob[pi];
  const int m0 = tile * kTcM;
  const int n0 = blockIdx.y * NTILE;
  const int K = args.k;
  const int kbeg = blockIdx.z * args.k_per_cta;
  const int kend = min(K, kbeg + args.k_per_cta);
  const int nchunks = max(0, (kend - kbeg + kTcKChunk - 1) / kTcKChunk);

  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < kTcStages; ++i) mbar_init(&sm.mbar[i], 1);
    fence_mbar_init();
    sm.timed_out = 0;
  }
  if (warp == 0) tmem_alloc(&sm.tmem_base, NTILE);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = sm.tmem_base;

  pdl_wait();  // x, row_gather and n_dev come from earlier kernels
  pdl_launch_dependents();
  const int n_live = args.n_dev ? min(args.n, *args.n_dev) : args.n;
  const uint32_t idesc = umma_idesc_f16(kTcM, NTILE);

  // Every thread copies the same (row, 16-byte column) pieces of every K chunk: work out their
  // source rows and shared-memory offsets once, so that a chunk costs one add and one cp.async
  // per piece (address arithmetic per piece per chunk used to dominate this kernel).
  constexpr int kAPieces = kTcM * 8 / kTcThreads, kBPieces = NTILE * 8 / kTcThreads;
  static_assert(kTcM * 8 % kTcThreads == 0 && NTILE * 8 % kTcThreads == 0, "pieces per thread");
  const __half* a_src[kAPieces];
  const __half* b_src[kBPieces];
  uint32_t a_off[kAPieces], b_off[kBPieces];
  uint32_t a_live = 0u, b_live = 0u;
  auto piece = [](int idx, int rows, int& row, int& c) {
    // a warp covers 8 rows x 4 chunks: 64 contiguous source bytes per row, and every 8
    // consecutive lanes write 128 contiguous shared-memory bytes
    const int r_lo = idx & 7, c_lo = (idx >> 3) & 3, rest = idx >> 5;
    c = ((rest & 1) << 2) | c_lo;
    row = ((rest >> 1) << 3) | r_lo;
    (void)rows;
  };
#pragma unroll
  for (int it = 0; it < kAPieces; ++it) {
    int row, c;
    piece(threadIdx.x + it * kTcThreads, kTcM, row, c);
    const int m = m0 + row;
    a_off[it] = static_cast<uint32_t>((c * kTcM + row) * 16);
    a_src[it] = pb.a;
    if (m < pb.m) {
      a_src[it] = pb.a + static_cast<size_t>(m) * K + kbeg + 8 * c;
      a_live |= 1u << it;
    }
  }
#pragma unroll
  for (int it = 0; it < kBPieces; ++it) {
    int row, c;
    piece(threadIdx.x + it * kTcThreads, NTILE, row, c);
    const int n = n0 + row;
    b_off[it] = static_cast<uint32_t>((c * NTILE + row) * 16);
    b_src[it] = args.x;
    if (n < n_live) {
      const int src = args.row_gather ? args.row_gather[n] : n;
      b_src[it] = args.x + static_cast<size_t>(src) * K + kbeg + 8 * c;
      b_live |= 1u << it;
    }
  }
  auto issue_chunk = [&](int i) {
    const int s = i % kTcStages;
    const int koff = i * kTcKChunk;  // halves from the start of this CTA's K range
#pragma unroll
    for (int it = 0; it < kAPieces; ++it) {
      const bool live = (a_live >> it) & 1u;
      cp_async_16(sm.a[s] + a_off[it], live ? a_src[it] + koff : a_src[it], live);
    }
#pragma unroll
    for (int it = 0; it < kBPieces; ++it) {
      const bool live = (b_live >> it) & 1u;
      cp_async_16(sm.b[s] + b_off[it], live ? b_src[it] + koff : b_src[it], live);
    }
  };

  // Software pipeline over the K chunks: copies run kTcStages-1 chunks ahead of the MMAs.
  uint32_t phase_bits = 0u;  // bit s = parity to wait for on mbar[s]
  bool ok = true;
#pragma unroll
  for (int i = 0; i < kTcStages - 1; ++i) {
    if (i < nchunks) issue_chunk(i);
    cp_async_commit();
  }
  for (int i = 0; i < nchunks; ++i) {
    const int s = i % kTcStages;
    cp_async_wait<kTcStages - 2>();  // this thread's copies of chunk i have landed
    fence_proxy_async();             // ... and are visible to the tensor core's reads
    __syncthreads();
    if (threadIdx.x == 0) {
      tcgen05_fence_after();
      const uint32_t a_addr = smem_u32(sm.a[s]), b_addr = smem_u32(sm.b[s]);
#pragma unroll
      for (int j = 0; j < kTcKChunk / 16; ++j) {
        const uint64_t da = umma_smem_desc(a_addr + j * 2 * kTcM * 16, kTcM * 16, 128);
        const uint64_t db = umma_smem_desc(b_addr + j * 2 * NTILE * 16, NTILE * 16, 128);
        umma_f16_ss(tmem, da, db, idesc, (i > 0 || j > 0) ? 1u : 0u);
      }
      umma_commit(&sm.mbar[s]);
    }
    // refill the stage that chunk i-1 used, once its MMAs have drained
    const int nxt = i + kTcStages - 1;
    if (nxt < nchunks) {
      if (i >= 1) {
        const int ps = (i - 1) % kTcStages;
        if (!mbar_wait_bounded(&sm.mbar[ps], (phase_bits >> ps) & 1u)) ok = false;
        phase_bits ^= 1u << ps;
      }
      issue_chunk(nxt);
    }
    cp_async_commit();
  }
  // drain: chunks up to nchunks - kTcStages - 1 were waited for when their stage was refilled
  for (int c = max(0, nchunks - kTcStages); c < nchunks; ++c) {
    const int s = c % kTcStages;
    if (!mbar_wait_bounded(&sm.mbar[s], (phase_bits >> s) & 1u)) ok = false;
    phase_bits ^= 1u << s;
  }
  if (!ok) sm.timed_out = 1;
  tcgen05_fence_after();
  __syncthreads();
  const bool failed = sm.timed_out != 0;

  tc_gemm_epilogue<NTILE>(args, pb, reinterpret_cast<float*>(smem_raw), tmem, failed, nchunks, m0, n0, n_live, cluster);
}

// ---- TMA-fed variant ------------------------------------------------------------------------
// Same tile, but the operands lie in shared memory in the 128-byte-swizzled K-major layout (8 rows x 128
// bytes per atom), so that a K chunk of an operand arrives with ONE tensor copy whose rows are 128
// contiguous bytes.  (Boxes of 16-byte rows that land in the no-swizzle core-matrix order made the copy
// engine the limit: 1536 requests per chunk; 16384 x 1024 x 256: 75 us.)  Rows past the matrix read as
// zeros.  One thread issues the copies (a full/empty mbarrier pair per stage), one thread the MMAs; all
// four warps run the epilogue.  The matrix chunks of the first stages are requested before the wait for
// the predecessor kernel when the caller says that they are older.  Used when the activation rows are not
// gathered (row_gather == nullptr).
struct TcTmaMaps {
  CUtensorMap a[3];
  CUtensorMap x;
};
constexpr int kTcRowBytes = kTcKChunk * 2;
static_assert(kTcRowBytes == 128, "one swizzle row per operand row and chunk");

// Stages of 64 columns: as many as let two CTAs share an SM, so that one's start and epilogue run under the other's products.
// With four stages of 128 rows there was one CTA to an SM, and the 256 CTAs of 16384 rows ran in two waves: 31.0 us at 1024 columns, now
// 16.8 (with the reads of an unsplit tile below).
constexpr int tma_stages(int ntile) { return ntile == 128 ? 3 : 4; }

// Parity of the last copy round of stage s when `issued` chunks went round-robin over `stages`, -1: none.
constexpr int last_round_parity(int issued, int s, int stages) { return issued > s ? ((issued - 1 - s) / stages) & 1 : -1; }
static_assert(last_round_parity(0, 0, 4) == -1 && last_round_parity(3, 2, 4) == 0 && last_round_parity(3, 3, 4) == -1 && last_round_parity(4, 3, 4) == 0, "first round");
static_assert(last_round_parity(5, 0, 4) == 1 && last_round_parity(5, 1, 4) == 0 && last_round_parity(8, 3, 4) == 1 && last_round_parity(9, 0, 4) == 0, "later rounds");
static_assert(last_round_parity(4, 0, 3) == 1 && last_round_parity(4, 1, 3) == 0 && last_round_parity(7, 0, 3) == 0 && last_round_parity(2, 2, 3) == -1, "three stages");

template <int NTILE>
struct TcTmaSmem {  // at a 1024-byte boundary
  static constexpr int kStages = tma_stages(NTILE);
  uint8_t a[kStages][kTcM * kTcRowBytes];
  uint8_t b[kStages][NTILE * kTcRowBytes];
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t done;
  uint32_t tmem_base;
  int32_t timed_out;
};

template <int NTILE>
__global__ void __launch_bounds__(kTcThreads) umma_gemm_tma_kernel(const __grid_constant__ TcGemmArgs args,
                                                                   const __grid_constant__ TcTmaMaps maps) {
  constexpr int kStages = tma_stages(NTILE);
  extern __shared__ uint4 smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>(smem_raw) + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  auto& sm = *reinterpret_cast<TcTmaSmem<NTILE>*>(base);
  cg::cluster_group cluster = cg::this_cluster();
  const int warp = warp_uniform(threadIdx.x >> 5);

  int tile = blockIdx.x, pi = 0;
  while (pi + 1 < args.num_problems && tile >= (args.prob[pi].m + kTcM - 1) / kTcM) {
    tile -= (args.prob[pi].m + kTcM - 1) / kTcM;
    ++pi;
  }
  const SkinnyProblem& pb = args.prob[pi];
  const int m0 = tile * kTcM;
  const int n0 = blockIdx.y * NTILE;
  const int K = args.k;
  const int kbeg = blockIdx.z * args.k_per_cta;
  const int kend = min(K, kbeg + args.k_per_cta);
  const int nchunks = max(0, (kend - kbeg + kTcKChunk - 1) / kTcKChunk);

  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], 1);
    }
    mbar_init(&sm.done, 1);
    fence_mbar_init();
    sm.timed_out = 0;
  }
  if (warp == 0) tmem_alloc(&sm.tmem_base, NTILE);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = warp_uniform(sm.tmem_base);
  constexpr uint32_t kBytes = (kTcM + NTILE) * kTcRowBytes;
  auto load_a = [&](int i) {
    const int s = i % kStages;
    mbar_arrive_expect_tx(&sm.full[s], kBytes);
    tma_load_2d(sm.a[s], &maps.a[pi], kbeg + i * kTcKChunk, m0, &sm.full[s]);
  };
  const int ahead = args.a_before_wait ? min(nchunks, kStages) : 0;
  if (threadIdx.x == 0)
    for (int i = 0; i < ahead; ++i) load_a(i);

  pdl_wait();  // x and n_dev come from earlier kernels
  pdl_launch_dependents();
  const int n_live = args.n_dev ? min(args.n, *args.n_dev) : args.n;

  int issued = 0;
  if (threadIdx.x == 0) {
    // producer: one tensor copy per operand per K chunk, kStages chunks in flight
    for (int i = 0; i < nchunks; ++i, ++issued) {
      const int s = i % kStages;
      if (i >= kStages && !mbar_wait_bounded(&sm.empty[s], ((i / kStages) - 1) & 1)) {
        sm.timed_out = 1;
        break;
      }
      if (i >= ahead) load_a(i);
      tma_load_2d(sm.b[s], &maps.x, kbeg + i * kTcKChunk, n0, &sm.full[s]);
    }
  }
  __syncwarp();
  if (warp == 1) {
    // consumer: four K = 16 MMAs per chunk; the commit frees the stage for the producer
    const uint32_t idesc = umma_idesc_f16(kTcM, NTILE);
    bool ok = true;
    for (int i = 0; i < nchunks; ++i) {
      const int s = i % kStages;
      ok = mbar_wait_warp(&sm.full[s], (i / kStages) & 1);
      if (!ok) break;
      tcgen05_fence_after();
      const uint64_t da = umma_smem_desc_sw128(smem_u32(sm.a[s])), db = umma_smem_desc_sw128(smem_u32(sm.b[s]));
      if (elect_one()) {
#pragma unroll
        for (int j = 0; j < kTcKChunk / 16; ++j) umma_f16_ss(tmem, da + 2 * j, db + 2 * j, idesc, (i > 0 || j > 0) ? 1u : 0u);
        umma_commit(&sm.empty[s]);
      }
    }
    if (elect_one()) {
      if (!ok) sm.timed_out = 1;
      umma_commit(&sm.done);  // arrives once every MMA issued so far has completed
    }
    __syncwarp();
  }
  if (!mbar_wait_bounded(&sm.done, 0)) sm.timed_out = 1;
  tcgen05_fence_after();
  __syncthreads();
  const bool failed = sm.timed_out != 0;
  if (failed && threadIdx.x == 0)  // copies in flight must not land in a buffer that is read as the partial tile
    for (int s = 0; s < kStages; ++s)
      if (last_round_parity(issued, s, kStages) >= 0) mbar_wait_bounded(&sm.full[s], last_round_parity(issued, s, kStages));
  __syncthreads();
  tc_gemm_epilogue<NTILE>(args, pb, reinterpret_cast<float*>(base), tmem, failed, nchunks, m0, n0, n_live, cluster);
}

// ---- tiles of 128 rows x 256 outputs ----------------------------------------------------------------
// With many rows the operands' way from L2 is what counts, and a tile of 128 outputs x 64 (128) rows asks for 24 (32) KB to do what this one
// does with 12 (24).  The rows are the M side, a whole matrix of the usual rank the N side; one CTA to an SM, four stages of 48 KB.  A lane
// of the accumulator is a row; the tile goes through shared memory (padded lines) to rows of 16-byte stores, or to the cluster's sums.
constexpr int kBigRows = 128, kBigOuts = 256, kBigThreads = 256, kBigStages = 4, kBigLine = kBigOuts + 4;  // floats of a line
struct TcBigMaps {
  CUtensorMap a[3];
  CUtensorMap x;
  int32_t outs[3];  // outputs of a tile: a multiple of 16, 256 at most
};
struct TcBigSmem {  // at a 1024-byte boundary
  uint8_t a[kBigStages][kBigOuts * kTcRowBytes];
  uint8_t x[kBigStages][kBigRows * kTcRowBytes];
  uint64_t full[kBigStages];
  uint64_t empty[kBigStages];
  uint64_t done;
  uint32_t tmem_base;
  int32_t timed_out;
};
static_assert(kBigRows * kBigLine * sizeof(float) <= sizeof(TcBigSmem::a) + sizeof(TcBigSmem::x), "the tile lies where the stages were");

// grid (tiles of outputs over all problems, row tiles, ksplit); cluster (1, 1, ksplit)
__global__ void __launch_bounds__(kBigThreads) umma_gemm_big_kernel(const __grid_constant__ TcGemmArgs args, const __grid_constant__ TcBigMaps maps) {
  extern __shared__ uint4 smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>(smem_raw) + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  auto& sm = *reinterpret_cast<TcBigSmem*>(base);
  cg::cluster_group cluster = cg::this_cluster();
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  int tile = blockIdx.x, pi = 0;
  while (pi + 1 < args.num_problems && tile >= (args.prob[pi].m + kBigOuts - 1) / kBigOuts) {
    tile -= (args.prob[pi].m + kBigOuts - 1) / kBigOuts;
    ++pi;
  }
  const SkinnyProblem& pb = args.prob[pi];
  const int outs = maps.outs[pi], m0 = tile * outs, n0 = blockIdx.y * kBigRows;
  const int kbeg = blockIdx.z * args.k_per_cta, kend = min(args.k, kbeg + args.k_per_cta);
  const int nchunks = max(0, (kend - kbeg + kTcKChunk - 1) / kTcKChunk);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kBigStages; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], 1);
    }
    mbar_init(&sm.done, 1);
    fence_mbar_init();
    sm.timed_out = 0;
  }
  if (warp == 0) tmem_alloc(&sm.tmem_base, kBigOuts);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = warp_uniform(sm.tmem_base);
  auto load_a = [&](int i) {
    const int s = i % kBigStages;
    mbar_arrive_expect_tx(&sm.full[s], (kBigRows + outs) * kTcRowBytes);
    tma_load_2d(sm.a[s], &maps.a[pi], kbeg + i * kTcKChunk, m0, &sm.full[s]);
  };
  const int ahead = args.a_before_wait ? min(nchunks, kBigStages) : 0;
  if (threadIdx.x == 0)
    for (int i = 0; i < ahead; ++i) load_a(i);

  pdl_wait();  // x and n_dev come from earlier kernels
  pdl_launch_dependents();
  const int n_live = args.n_dev ? min(args.n, *args.n_dev) : args.n;

  int issued = 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < nchunks; ++i, ++issued) {
      const int s = i % kBigStages;
      if (i >= kBigStages && !mbar_wait_bounded(&sm.empty[s], ((i / kBigStages) - 1) & 1)) {
        sm.timed_out = 1;
        break;
      }
      if (i >= ahead) load_a(i);
      tma_load_2d(sm.x[s], &maps.x, kbeg + i * kTcKChunk, n0, &sm.full[s]);
    }
  }
  __syncwarp();
  if (warp == 1) {
    const uint32_t idesc = umma_idesc_f16(kBigRows, outs);
    bool ok = true;
    for (int i = 0; i < nchunks; ++i) {
      const int s = i % kBigStages;
      ok = mbar_wait_warp(&sm.full[s], (i / kBigStages) & 1);
      if (!ok) break;
      tcgen05_fence_after();
      const uint64_t dx = umma_smem_desc_sw128(smem_u32(sm.x[s])), da = umma_smem_desc_sw128(smem_u32(sm.a[s]));
      if (elect_one()) {
#pragma unroll
        for (int j = 0; j < kTcKChunk / 16; ++j) umma_f16_ss(tmem, dx + 2 * j, da + 2 * j, idesc, (i > 0 || j > 0) ? 1u : 0u);
        umma_commit(&sm.empty[s]);
      }
    }
    if (elect_one()) {
      if (!ok) sm.timed_out = 1;
      umma_commit(&sm.done);  // arrives once every MMA issued so far has completed
    }
    __syncwarp();
  }
  if (!mbar_wait_bounded(&sm.done, 0)) sm.timed_out = 1;
  tcgen05_fence_after();
  __syncthreads();
  const bool failed = sm.timed_out != 0;
  if (failed && threadIdx.x == 0)  // copies in flight must not land in a buffer that is read as the tile
    for (int s = 0; s < kBigStages; ++s)
      if (last_round_parity(issued, s, kBigStages) >= 0) mbar_wait_bounded(&sm.full[s], last_round_parity(issued, s, kBigStages));
  __syncthreads();

  // accumulator -> lines of shared memory: warp w rows 32 (w % 4) .. + 31, half w / 4 of the outputs
  float* part = reinterpret_cast<float*>(base);
  float* line = part + (32 * (warp & 3) + lane) * kBigLine;
  const int half = kBigOuts / 2 * (warp >> 2);
  if (!failed && nchunks > 0) {
    const uint32_t at = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll 1
    for (int c0 = half; c0 < min(outs, half + kBigOuts / 2); c0 += 16) {
      float v[16];
      tmem_ld_16(at + c0, v);
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(line + c0 + 4 * j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
  } else {
    for (int c = half; c < half + kBigOuts / 2; ++c) line[c] = 0.f;
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kBigOuts);
  if (failed && threadIdx.x == 0 && args.status) atomicExch(args.status, TRIS_ERR_TIMEOUT);
  cluster.sync();
  // every CTA of the cluster adds up and stores its own rows, a warp eight outputs a lane of one row at a time
  const int nblk = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int per = (kBigRows + nblk - 1) / nblk, r_end = min(kBigRows, (rank + 1) * per), m = m0 + 8 * lane;
  const bool lives = 8 * lane < outs && m < pb.m;
  const bool whole = m + 8 <= pb.m && pb.m % 8 == 0 && (reinterpret_cast<uintptr_t>(pb.out) & 15u) == 0;
  const float* parts[8];
#pragma unroll
  for (int b = 0; b < 8; ++b) parts[b] = cluster.map_shared_rank(part, b < nblk ? b : 0) + 8 * lane;
#pragma unroll 2
  for (int r = rank * per + warp; r < r_end; r += kBigThreads / 32) {
    const int n = n0 + r;
    if (n >= n_live || !lives) continue;
    float v[8] = {};
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      if (b >= nblk) break;
      const float4 lo = *reinterpret_cast<const float4*>(parts[b] + r * kBigLine), hi = *reinterpret_cast<const float4*>(parts[b] + r * kBigLine + 4);
      v[0] += lo.x, v[1] += lo.y, v[2] += lo.z, v[3] += lo.w, v[4] += hi.x, v[5] += hi.y, v[6] += hi.z, v[7] += hi.w;
    }
    const size_t at = static_cast<size_t>(n) * pb.m + m;
    if (whole && pb.out_mode == TRIS_OUT_F32) {
      float4* dst = reinterpret_cast<float4*>(static_cast<float*>(pb.out) + at);
      dst[0] = make_float4(v[0], v[1], v[2], v[3]);
      dst[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else if (whole && pb.out_mode == TRIS_OUT_F16) {
      *reinterpret_cast<uint4*>(static_cast<__half*>(pb.out) + at) =
          make_uint4(h2_as_u32(__floats2half2_rn(v[0], v[1])), h2_as_u32(__floats2half2_rn(v[2], v[3])), h2_as_u32(__floats2half2_rn(v[4], v[5])), h2_as_u32(__floats2half2_rn(v[6], v[7])));
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (m + j >= pb.m) continue;
        if (pb.out_mode == TRIS_OUT_F32) static_cast<float*>(pb.out)[at + j] = v[j];
        else static_cast<__half*>(pb.out)[static_cast<size_t>(n) * pb.m + out_mode_pos(m + j, pb.out_mode)] = __float2half_rn(v[j]);
      }
    }
  }
  cluster.sync();  // keep every CTA's shared memory alive until its peers have read it
}

static int launch_umma_big(const TcGemmArgs& args, const TcBigMaps& maps, int tiles, int ksplit, cudaStream_t stream, bool pdl) {
  constexpr size_t smem = sizeof(TcBigSmem) + 1024;
  static_assert(smem <= 227 * 1024, "shared memory");
  static bool configured[64] = {};
  int dev = 0;
  TRIS_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    TRIS_CUDA(cudaFuncSetAttribute(umma_gemm_big_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  return check_cuda(launch_kernel(umma_gemm_big_kernel, dim3(tiles, ceil_div(args.n, kBigRows), ksplit), dim3(kBigThreads), smem, stream, pdl, ksplit, args, maps),
                    "umma_gemm_big_kernel launch");
}

template <int NTILE>
static int launch_umma(const TcGemmArgs& args, int mtiles, int ksplit, cudaStream_t stream, bool pdl) {
  const size_t smem = std::max(sizeof(TcSmem<NTILE>), static_cast<size_t>(NTILE) * kTcM * 4 + 128);
  static bool configured[64] = {};
  int dev = 0;
  TRIS_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    TRIS_CUDA(cudaFuncSetAttribute(umma_gemm_kernel<NTILE>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  return check_cuda(launch_kernel(umma_gemm_kernel<NTILE>, dim3(mtiles, ceil_div(args.n, NTILE), ksplit),
                                  dim3(kTcThreads), smem, stream, pdl, ksplit, args),
                    "umma_gemm_kernel launch");
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda).
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
  static std::atomic<void*> cached{nullptr};
  static std::atomic<bool> tried{false};
  if (!tried.load(std::memory_order_acquire)) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      fn = nullptr;
    cudaGetLastError();
    cached.store(fn, std::memory_order_release);
    tried.store(true, std::memory_order_release);
  }
  return reinterpret_cast<EncodeTiledFn>(cached.load(std::memory_order_acquire));
}

bool encode_rows_map(CUtensorMap* map, const void* base, int rows, int cols, int stride, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr || rows <= 0) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(stride) * 2};  // bytes, dimension 1
  const cuuint32_t box[2] = {kTcKChunk, static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NTILE>
static int launch_umma_tma(const TcGemmArgs& args, const TcTmaMaps& maps, int mtiles, int ksplit, cudaStream_t stream,
                           bool pdl) {
  const size_t smem = std::max(sizeof(TcTmaSmem<NTILE>), static_cast<size_t>(NTILE) * kTcM * 4) + 1024;
  static bool configured[64] = {};
  int dev = 0;
  TRIS_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    TRIS_CUDA(cudaFuncSetAttribute(umma_gemm_tma_kernel<NTILE>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  return check_cuda(launch_kernel(umma_gemm_tma_kernel<NTILE>, dim3(mtiles, ceil_div(args.n, NTILE), ksplit),
                                  dim3(kTcThreads), smem, stream, pdl, ksplit, args, maps),
                    "umma_gemm_tma_kernel launch");
}

// True when the tensor-core path applies: more rows than the skinny GEMM takes better for a dense contraction, K a multiple
// of the 64-column chunk, 16-byte aligned rows.
bool tc_gemm_applicable(int n, int k, const __half* x, const SkinnyProblem* probs, int num_problems) {
  if (n <= 32 || (k % kTcKChunk) != 0 || (reinterpret_cast<uintptr_t>(x) & 15u)) return false;
  for (int i = 0; i < num_problems; ++i)
    if (reinterpret_cast<uintptr_t>(probs[i].a) & 15u) return false;
  return true;
}

constexpr int kTcSms = 148;
// Split K over the cluster until the GPU is full or a CTA would get fewer than two 64-column chunks: a CTA's
// time is its chain of chunk loads and MMAs, so shorter chains win (measured at 128 and 1024 rows: 85.7 us
// per layer with a floor of two chunks, 86.8 with four; a cluster of 16 is slower again)
static int column_split(int tiles, int k) {
  int ksplit = 1;
  while (ksplit < 8 && tiles * ksplit < kTcSms && k / (ksplit * 2) >= 2 * kTcKChunk) ksplit *= 2;
  return ksplit;
}
// Clusters of 1, 2, 4 and 8 CTAs that a B200 holds at once where two of the CTAs share an SM and where one has it to itself: SMs come in
// groups of 16 to 20, and a cluster does not span two (cudaOccupancyMaxActiveClusters for kernels of this footprint).
static int clusters_at_once(bool alone, int ksplit) {
  constexpr int kClusters[2][4] = {{296, 148, 71, 33}, {148, 74, 33, 15}};
  return kClusters[alone][ksplit >= 8 ? 3 : ksplit >> 1];
}
// 128-row tiles re-read the matrices half as often; 64-row tiles give a small batch more CTAs.  For long rows, where the
// operands' way from L2 is what counts, fewer 128-row tiles do too, if the split of the columns fills the GPU all the same: us,
// 64-row / 128-row tiles of 256 outputs, 8192 columns, 40 tiles of 128 rows 22.4 / 21.8, 74: 43.2 / 35.0; 14336 columns, 24:
// 23.7 / 21.7, 40: 38.5 / 31.7, 74: 74.9 / 56.3 (at 4096 columns 12.6 / 14.4).  Eighths of 8192 columns are too short for it (19 to
// 32 tiles 0.92 to 1.06 of the time; of 10240, 0.92 to 1.02).  And if the clusters run at once: 72 of four CTAs, of which 71 fit,
// 28.4 / 40.6, 34 of eight, of which 33 fit, 17.6 / 27.2.  Gathered 128-row tiles (128 KB) have an SM to themselves, and two turns of
// them are no longer than one of 64-row tiles that share it (8192 columns, 30 tiles 66 / 56; 32 tiles, a third turn, 66 / 80).
static int rows_per_tile(int mtiles, int n, int k, bool gathered) {
  const int tiles128 = mtiles * ceil_div(n, 128), split128 = column_split(tiles128, k);
  // as many as SMs: twice as many of 64 rows run at once too, and two to an SM hide each other's start (us, 64 / 128: 9472 x 1024 x 256
  // 13.4 / 14.7, 9472 x 8192 x 256 54.2 / 60.4; with one more tile 20.4 / 15.5)
  if (tiles128 >= kTcSms) return tiles128 == kTcSms && !gathered ? 64 : 128;
  if (tiles128 * 8 < kTcSms || k < (split128 == 8 && !gathered ? 10240 : 8192)) return 64;
  if (tiles128 <= (gathered ? 2 : 1) * clusters_at_once(gathered, split128)) return 128;
  const int tiles64 = mtiles * ceil_div(n, 64);
  return tiles64 <= clusters_at_once(false, column_split(tiles64, k)) ? 64 : 128;  // neither runs at once: 36 tiles, 0.9 to 1.0 of the time
}

// Split of the columns for tiles of 128 rows x 256 outputs, 0: smaller tiles are better.  A CTA fills 192 KB of stages before its first product and a
// 133 KB tile goes through shared memory after its last one, which takes many rows to pay; in a layer's sequence half of that start runs under the
// kernel before, which is where they are used.  us, smaller tiles / these, launch by launch: two matrices of 256 x 2048 and a router of 64, 1700 rows
// 13.7 / 14.6, 2048 18.2 / 14.4 (halves of the columns), of 256 x 4096 and a router of 8, 1300, 1700 and 2048 rows 20.9 / 18.5, 22.6 / 19.0,
// 30.4 / 19.2; 256 x 1024, 4072, 6144, 12000 and 16384 rows 10.3 / 11.8, 13.0 / 11.8, 16.5 / 12.2, 17.2 / 12.6; 320 x 1024 in tiles of 160 outputs,
// 3600, 4072, 8192 and 16384 rows 13.4 / 13.6, 13.5 / 9.8, 19.2 / 10.1, 33.2 / 19.5 (in tiles of 256 and 64 8192 rows 12.4, 16384 23.0); 128 x 1024,
// 8192 and 12000 10.2 / 10.3, 12.8 / 10.5; 256 x 14336, 2048, 3000 and 4072 rows 24.7 / 28.5, 35.0 / 33.6, 39.4 / 38.6.  Parts of fewer than
// 1024 columns are not worth the sum (1024 columns, 6144 rows 12.0), nor are eighths (blocks whose down backbone has 1280 and 1600 rows of 14336
// columns 127 / 132, 131 / 136).  Where the lines for split columns lie: 320 x 14336, 2758 rows (55) 36.5 / 43.6, 3600 rows 58.3 / 45.7; blocks with
// it, 1340, 1400 and 1460 tokens (gate and up in these tiles in all three; 52, 55 and 57 of down's) 1.015, 1.005 and 1.04; blocks with
// 128 x 14336, 1862, 1906 and 1950 tokens (58, 60, 62) 0.98, 0.99, 1.02.  Quarters of 1024 columns: two matrices of 256 x 4096, 1100 rows
// (73) 0.99 of a block, 1379 (89) 1.02.
static int big_tile_split(const SkinnyProblem* probs, int num_problems, int n, int k) {
  const int row_tiles = ceil_div(n, kBigRows);
  int tiles = 0, outs = 0, widest = 0;
  for (int i = 0; i < num_problems; ++i) {
    tiles += ceil_div(probs[i].m, kBigOuts) * row_tiles;
    outs += probs[i].m;
    widest = std::max(widest, probs[i].m);
  }
  int ksplit = 1;
  while (ksplit < 4 && tiles <= clusters_at_once(true, 2 * ksplit) && k / (ksplit * 2) >= 1024) ksplit *= 2;
  const int ctas = tiles * ksplit, filled = static_cast<int>(static_cast<long long>(outs) * row_tiles * ksplit / kBigOuts);  // tiles' worth of outputs
  if (ctas > kTcSms && ctas * 5 < ceil_div(ctas, kTcSms) * kTcSms * 4) return 0;
  if (ksplit == 1) return filled >= 40 ? 1 : 0;
  const int part = k / ksplit;
  const int least = part >= 3072 ? (widest <= 128 ? 62 : 57) : part >= 2048 ? 55 : (ksplit == 4 ? 85 : 70);
  return ctas >= 80 && filled >= least ? ksplit : 0;
}

int launch_tc_gemm(const SkinnyProblem* probs, int num_problems, const __half* x, const int32_t* row_gather, int n,
                   int k, cudaStream_t stream, bool pdl, const int32_t* n_dev, int32_t* status, bool a_before_wait) {
  TcGemmArgs args{};
  int mtiles = 0;
  for (int i = 0; i < num_problems; ++i) {
    args.prob[i] = probs[i];
    mtiles += ceil_div(probs[i].m, kTcM);
  }
  args.num_problems = num_problems;
  args.x = x;
  args.row_gather = row_gather;
  args.n_dev = n_dev;
  args.status = status;
  args.n = n;
  args.k = k;
  args.a_before_wait = pdl && a_before_wait;
  const int big = pdl && row_gather == nullptr ? big_tile_split(probs, num_problems, n, k) : 0;
  if (big > 0) {
    TcBigMaps maps;
    int tiles = 0;
    bool ok = encode_rows_map(&maps.x, x, n, k, k, kBigRows);
    for (int i = 0; i < num_problems && ok; ++i) {
      const int parts = ceil_div(probs[i].m, kBigOuts);
      maps.outs[i] = ceil_div(ceil_div(probs[i].m, parts), 16) * 16;  // equal tiles: 320 outputs are two of 160
      tiles += parts;
      ok = encode_rows_map(&maps.a[i], probs[i].a, probs[i].m, k, k, maps.outs[i]);
    }
    args.k_per_cta = ceil_div(ceil_div(k, big), kTcKChunk) * kTcKChunk;
    if (ok) return launch_umma_big(args, maps, tiles, big, stream, pdl);
  }
  const int ntile = rows_per_tile(mtiles, n, k, row_gather != nullptr);
  const int ntiles = ceil_div(n, ntile), ksplit = column_split(mtiles * ntiles, k);
  args.k_per_cta = ceil_div(ceil_div(k, ksplit), kTcKChunk) * kTcKChunk;
  if (row_gather == nullptr) {  // operands by tensor copies
    TcTmaMaps maps;
    bool ok = encode_rows_map(&maps.x, x, n, k, k, ntile);
    for (int i = 0; i < num_problems && ok; ++i) ok = encode_rows_map(&maps.a[i], probs[i].a, probs[i].m, k, k, kTcM);
    if (ok) {
      if (ntile == 64) return launch_umma_tma<64>(args, maps, mtiles, ksplit, stream, pdl);
      return launch_umma_tma<128>(args, maps, mtiles, ksplit, stream, pdl);
    }
  }
  if (ntile == 64) return launch_umma<64>(args, mtiles, ksplit, stream, pdl);
  return launch_umma<128>(args, mtiles, ksplit, stream, pdl);
}

}  // namespace tris
