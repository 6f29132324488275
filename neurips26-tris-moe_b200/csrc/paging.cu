// Streaming loader: gathers the payload blocks of the experts a batch routes to from pinned
// host memory into device staging slots.  The copy is a kernel that reads the (device-mapped)
// host buffers directly, so the set of active experts never has to travel to the host: the
// launch is enqueued on a side stream right after the route kernel and ordered with events.
#include <algorithm>

#include "common.cuh"

namespace tris {

struct PageArgs {
  TrisPageJob jobs[TRIS_MAX_PAGE_JOBS];
  int32_t num_jobs;
  const int32_t* expert_ids;
  const int32_t* num_segments_dev;
  int32_t num_segments;
  int32_t num_experts;
  int32_t* slot_table;
};

// CTAs of a pager and their warps.  The reads in flight have to cover the host link's latency, and the warps of coded pages keep up with it
// while they decode, on SMs that are not all as near to the link and of which a pager that starts beside another kernel gets
// fewer than there are; but no more of them: what is queued beyond that delays every other read of the memory system and every
// launch, and the kernels that work on what is there already run beside the pager.  With all warps of a page resident at once they took
// three times as long.  us, two streamed layers of 102 experts, nine states, 64 / 96 / 148 / 222 CTAs of coded pages: 538-600, 425-457,
// 354-369, 373-397; uncoded ones, whose threads have eight reads in flight, one layer, 20 / 28 / 64 / 148 CTAs: 590, 583, 583, 584, and 4
// tokens of 64 experts 205, 206, 209, 213.
constexpr int kPageWarps = 4, kPageThreads = 32 * kPageWarps, kPagerCtas = 32, kCodedPagerCtas = 148;

// Pieces of 16 KB (eight 16-byte reads a thread) of the active experts' blocks, dealt to the CTAs in turn.
__global__ void __launch_bounds__(kPageThreads) page_experts_kernel(const __grid_constant__ PageArgs args) {
  constexpr int kPiece = 8 * kPageThreads;  // 16-byte words
  const int nseg = args.num_segments_dev ? min(*args.num_segments_dev, args.num_segments) : args.num_segments;
  int per_segment = 0;
  for (int j = 0; j < args.num_jobs; ++j) per_segment += static_cast<int>(((args.jobs[j].bytes_per_expert >> 4) + kPiece - 1) / kPiece);
  for (int i = blockIdx.x; i < nseg * per_segment; i += gridDim.x) {
    const int seg = i / per_segment, e = args.expert_ids[seg];
    if (e < 0 || e >= args.num_experts) continue;
    int piece = i - seg * per_segment, j = 0;
    if (piece == 0 && threadIdx.x == 0) args.slot_table[e] = seg;
    for (;; ++j) {
      const int pieces = static_cast<int>(((args.jobs[j].bytes_per_expert >> 4) + kPiece - 1) / kPiece);
      if (piece < pieces) break;
      piece -= pieces;
    }
    const TrisPageJob& job = args.jobs[j];
    const long long vecs = job.bytes_per_expert >> 4, at = static_cast<long long>(piece) * kPiece + threadIdx.x;
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const char*>(job.host_src) + e * job.bytes_per_expert) + at;
    uint4* dst = reinterpret_cast<uint4*>(static_cast<char*>(job.dst) + seg * job.bytes_per_expert) + at;
    uint4 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (at + k * kPageThreads < vecs) v[k] = __ldcs(src + k * kPageThreads);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (at + k * kPageThreads < vecs) dst[k * kPageThreads] = v[k];
  }
}

// ---- coded pages -------------------------------------------------------------------------------------
// The grouping bitmap of a projection has a tenth of its bits set, and the host link is what a streamed layer waits
// for: 20 MB of raw bitmaps for two layers of 102 active experts take 360 us of 580.  A block of 1024 bytes is coded as
// the gaps between its ones, four bits each: 0 .. 14 zeros and a one, or 15 zeros and no one.  At one bit in ten that is
// 0.50 bits per bit, 7 % over the entropy (three or five bits: 0.58, 0.52), and, unlike the Golomb-Rice codes of the
// resident format (0.48 and a 0.25-bit index of sub-streams), any 16 bytes of it can be read without the ones before: a lane adds
// up what its symbols advance by, a warp scan gives it its place.  A block that would not get smaller stays as it is.
constexpr int kPageBlock = TRIS_PAGE_BLOCK_BYTES, kPageWords = kPageBlock / 4, kPageUnits = kPageBlock / 16;
static_assert(kPageUnits == 64 && kPageWords == 8 * 32, "two 16-byte words and eight 4-byte words a lane");

struct CodedPageArgs {
  TrisCodedPageJob jobs[TRIS_MAX_PAGE_JOBS];
  int32_t num_jobs;
  const int32_t* expert_ids;
  const int32_t* num_segments_dev;
  int32_t num_segments;
  int32_t num_experts;
  int32_t* slot_table;
};

__device__ __forceinline__ int symbols_advance(uint32_t w) {  // sum over eight symbols of the bits they stand for
  const uint32_t bytes = (w & 0x0F0F0F0Fu) + ((w >> 4) & 0x0F0F0F0Fu), skips = w & (w >> 1) & (w >> 2) & (w >> 3) & 0x11111111u;
  return static_cast<int>(__dp4a(bytes, 0x01010101u, 0u)) + 8 - __popc(skips);
}

// A load that stays where it is written: the next block is asked for before the last one is decoded.
__device__ __forceinline__ uint4 load_now(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.cs.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
// A warp decodes blocks dealt to it in turn, and asks for the next one before it decodes the last.
__global__ void __launch_bounds__(kPageThreads) page_coded_kernel(const __grid_constant__ CodedPageArgs args) {
  // the lanes' places in a block are some eight words apart: a pad word after every 32 keeps them out of one another's banks
  __shared__ uint32_t bits[kPageWarps][kPageWords + kPageWords / 32];
  __shared__ __align__(16) uint32_t code[kPageWarps][kPageWords];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nseg = args.num_segments_dev ? min(*args.num_segments_dev, args.num_segments) : args.num_segments;
  auto blocks_of = [&](int j) { return static_cast<int>((args.jobs[j].bytes_per_expert + kPageBlock - 1) / kPageBlock); };
  int per_segment = 0;
  for (int j = 0; j < args.num_jobs; ++j) per_segment += blocks_of(j);
  const int total = nseg * per_segment, step = gridDim.x * kPageWarps;
  const uint4 skip = make_uint4(~0u, ~0u, ~0u, ~0u);
  struct Block {
    uint4 a, b;
    uint4* dst;
    int units, left;  // 16-byte words of the code and of the block; -1: nothing to do
  };
  auto fetch = [&](int i) {
    Block f;
    f.left = -1;
    if (i >= total) return f;
    const int seg = i / per_segment, e = args.expert_ids[seg];
    if (e < 0 || e >= args.num_experts) return f;
    int block = i - seg * per_segment, j = 0;
    if (block == 0 && lane == 0) args.slot_table[e] = seg;
    for (; block >= blocks_of(j); ++j) block -= blocks_of(j);
    const TrisCodedPageJob& job = args.jobs[j];
    const int32_t* offset = job.block_offsets + static_cast<size_t>(e) * blocks_of(j) + block;
    const int first = offset[0];
    f.units = min(offset[1] - first, kPageUnits);
    const uint4* src = static_cast<const uint4*>(job.host_src) + first;
    f.a = f.b = skip;
    if (lane < f.units) f.a = load_now(src + lane);
    if (lane + 32 < f.units) f.b = load_now(src + lane + 32);
    f.left = static_cast<int>(min(static_cast<long long>(kPageBlock), job.bytes_per_expert - static_cast<long long>(block) * kPageBlock)) >> 4;
    f.dst = reinterpret_cast<uint4*>(static_cast<char*>(job.dst) + static_cast<size_t>(seg) * job.bytes_per_expert + static_cast<size_t>(block) * kPageBlock);
    return f;
  };
  int i = blockIdx.x * kPageWarps + warp;
  Block next = fetch(i);
#pragma unroll 1
  for (; i < total; i += step) {
    const Block f = next;
    next = fetch(i + step);
    if (f.left < 0) continue;
    if (f.units == kPageUnits) {
      if (lane < f.left) f.dst[lane] = f.a;
      if (lane + 32 < f.left) f.dst[lane + 32] = f.b;
      continue;
    }
    // The code's words are dealt to the lanes in runs of equal length, so that every lane has its share of the symbols.
    uint32_t* out = bits[warp];
    for (int q = lane; q < kPageWords + kPageWords / 32; q += 32) out[q] = 0u;
    uint4* in = reinterpret_cast<uint4*>(code[warp]);
    in[lane] = f.a;
    in[lane + 32] = f.b;
    __syncwarp();
    const int run = (4 * f.units + 31) >> 5, begin = lane * run, end = min(begin + run, 4 * f.units);
    int mine = 0;
    for (int q = begin; q < end; ++q) mine += symbols_advance(code[warp][q]);
    int upto = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xFFFFFFFFu, upto, o);
      if (lane >= o) upto += n;
    }
    int pos = upto - mine;
    for (int q = begin; q < end; ++q) {
      uint32_t w = code[warp][q];
#pragma unroll
      for (int k = 0; k < 8; ++k, w >>= 4) {
        const int gap = static_cast<int>(w & 15u), bit = pos + gap;
        if (gap != 15 && bit < 8 * kPageBlock) atomicOr(&out[(bit >> 5) + (bit >> 10)], 1u << (bit & 31));
        pos = bit + (gap != 15);
      }
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int q = lane + 32 * h;
      const uint32_t* w = out + 4 * q + (q >> 3);
      if (q < f.left) f.dst[q] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    __syncwarp();  // before the next block's zeros
  }
}

// One warp per block: its size in 16-byte units (offsets null) or its code.
__global__ void __launch_bounds__(32 * kPageWarps) code_blocks_kernel(const char* src, long long bytes_per_expert, int blocks, long long total, int32_t* units_out,
                                                                      const int32_t* offsets, uint4* dst) {
  __shared__ __align__(16) uint32_t code[kPageWarps][kPageWords];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long at = blockIdx.x * static_cast<long long>(kPageWarps) + warp;
  if (at >= total) return;
  const long long e = at / blocks, block = at - e * blocks;
  const int left = static_cast<int>(min(static_cast<long long>(kPageBlock), bytes_per_expert - block * kPageBlock)) >> 4;
  const uint4* from = reinterpret_cast<const uint4*>(src + e * bytes_per_expert + block * kPageBlock);
  uint32_t w[8];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint4 v = 2 * lane + h < left ? from[2 * lane + h] : make_uint4(0u, 0u, 0u, 0u);
    w[4 * h] = v.x, w[4 * h + 1] = v.y, w[4 * h + 2] = v.z, w[4 * h + 3] = v.w;
  }
  int last = -1;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (w[i]) last = (8 * lane + i) * 32 + 31 - __clz(w[i]);
  int before = last;  // last one up to this lane, then of the lanes before it
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xFFFFFFFFu, before, o);
    if (lane >= o) before = max(before, n);
  }
  before = __shfl_up_sync(0xFFFFFFFFu, before, 1);
  if (lane == 0) before = -1;
  auto walk = [&](auto symbol) {  // symbol(gap) for every one of this lane
    int prev = before;
#pragma unroll 1
    for (int i = 0; i < 8; ++i) {
      uint32_t v = i == 0 ? w[0] : i == 1 ? w[1] : i == 2 ? w[2] : i == 3 ? w[3] : i == 4 ? w[4] : i == 5 ? w[5] : i == 6 ? w[6] : w[7];
      for (; v; v &= v - 1) {
        const int pos = (8 * lane + i) * 32 + __ffs(v) - 1;
        symbol(pos - prev - 1);
        prev = pos;
      }
    }
  };
  int count = 0;
  walk([&](int gap) { count += gap / 15 + 1; });
  int upto = count;
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xFFFFFFFFu, upto, o);
    if (lane >= o) upto += n;
  }
  const int all = __shfl_sync(0xFFFFFFFFu, upto, 31), units = min((all + 31) / 32, kPageUnits);
  if (offsets == nullptr) {
    if (lane == 0) units_out[at] = units;
    return;
  }
  dst += offsets[at];
  if (units == kPageUnits) {
#pragma unroll
    for (int h = 0; h < 2; ++h) dst[2 * lane + h] = make_uint4(w[4 * h], w[4 * h + 1], w[4 * h + 2], w[4 * h + 3]);
    return;
  }
  uint4* out = reinterpret_cast<uint4*>(code[warp]);
  out[lane] = out[lane + 32] = make_uint4(~0u, ~0u, ~0u, ~0u);  // what is left of the last unit: skips
  __syncwarp();
  int to = upto - count;
  walk([&](int gap) {
    to += gap / 15;
    atomicAnd(&code[warp][to >> 3], ~((15u ^ static_cast<uint32_t>(gap % 15)) << (4 * (to & 7))));
    ++to;
  });
  __syncwarp();
  if (lane < units) dst[lane] = out[lane];
  if (lane + 32 < units) dst[lane + 32] = out[lane + 32];
}

}  // namespace tris

using namespace tris;

extern "C" int tris_page_code_blocks(const void* src_dev, int64_t bytes_per_expert, int32_t num_experts, int32_t* units_out, const int32_t* block_offsets,
                                     void* dst, void* stream) {
  TRIS_REQUIRE(src_dev && (block_offsets ? dst != nullptr : units_out != nullptr), TRIS_ERR_INVALID_ARG, "tris_page_code_blocks: null pointer");
  TRIS_REQUIRE(bytes_per_expert > 0 && (bytes_per_expert & 15) == 0 && num_experts >= 0, TRIS_ERR_INVALID_ARG, "tris_page_code_blocks: bad sizes");
  TRIS_REQUIRE(((reinterpret_cast<uintptr_t>(src_dev) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0, TRIS_ERR_INVALID_ARG,
               "tris_page_code_blocks: buffers must be 16-byte aligned");
  const long long blocks = (bytes_per_expert + kPageBlock - 1) / kPageBlock, total = blocks * num_experts;
  TRIS_REQUIRE(total * kPageUnits <= 0x7FFFFFFFll, TRIS_ERR_UNSUPPORTED, "tris_page_code_blocks: more than 2^31 16-byte units");
  if (total == 0) return TRIS_OK;
  if (block_offsets) {  // pinned host memory: by its address on the device
    cudaPointerAttributes at{};
    TRIS_CUDA(cudaPointerGetAttributes(&at, dst));
    TRIS_REQUIRE(at.type != cudaMemoryTypeUnregistered, TRIS_ERR_INVALID_ARG, "tris_page_code_blocks: the code needs device memory or pinned host memory");
    if (at.type == cudaMemoryTypeHost) dst = at.devicePointer;
  }
  code_blocks_kernel<<<static_cast<unsigned>((total + kPageWarps - 1) / kPageWarps), 32 * kPageWarps, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const char*>(src_dev), bytes_per_expert, static_cast<int>(blocks), total, units_out, block_offsets, static_cast<uint4*>(dst));
  return check_cuda(cudaGetLastError(), "code_blocks_kernel launch");
}

int tris::page_coded_experts_impl(const TrisCodedPageJob* jobs, int num_jobs, const int32_t* expert_ids, const int32_t* num_segments_dev,
                                  int num_segments, int num_experts, int32_t* slot_table, bool reset, cudaStream_t stream) {
  TRIS_REQUIRE(jobs && expert_ids && slot_table, TRIS_ERR_INVALID_ARG, "tris_page_coded_experts: null pointer");
  TRIS_REQUIRE(num_jobs >= 1 && num_jobs <= TRIS_MAX_PAGE_JOBS, TRIS_ERR_INVALID_ARG,
               "tris_page_coded_experts: %d jobs (1..%d supported)", num_jobs, TRIS_MAX_PAGE_JOBS);
  TRIS_REQUIRE(num_segments >= 0 && num_experts > 0, TRIS_ERR_INVALID_ARG, "tris_page_coded_experts: bad sizes");
  if (num_segments == 0) return TRIS_OK;
  CodedPageArgs args{};
  for (int j = 0; j < num_jobs; ++j) {
    TRIS_REQUIRE(jobs[j].host_src && jobs[j].block_offsets && jobs[j].dst && jobs[j].bytes_per_expert > 0 && (jobs[j].bytes_per_expert & 15) == 0,
                 TRIS_ERR_INVALID_ARG, "tris_page_coded_experts: job %d needs pointers and a block size that is a multiple of 16", j);
    TRIS_REQUIRE(((reinterpret_cast<uintptr_t>(jobs[j].host_src) | reinterpret_cast<uintptr_t>(jobs[j].dst)) & 15) == 0,
                 TRIS_ERR_INVALID_ARG, "tris_page_coded_experts: job %d buffers must be 16-byte aligned", j);
    args.jobs[j] = jobs[j];
    void* dev_alias = nullptr;  // as for uncoded pages
    TRIS_CUDA(cudaHostGetDevicePointer(&dev_alias, const_cast<void*>(jobs[j].host_src), 0));
    args.jobs[j].host_src = dev_alias;
  }
  args.num_jobs = num_jobs;
  args.expert_ids = expert_ids;
  args.num_segments_dev = num_segments_dev;
  args.num_segments = num_segments;
  args.num_experts = num_experts;
  args.slot_table = slot_table;
  if (reset) TRIS_CUDA(cudaMemsetAsync(slot_table, 0xFF, sizeof(int32_t) * static_cast<size_t>(num_experts), stream));
  page_coded_kernel<<<kCodedPagerCtas, kPageThreads, 0, stream>>>(args);
  return check_cuda(cudaGetLastError(), "page_coded_kernel launch");
}
extern "C" int tris_page_coded_experts(const TrisCodedPageJob* jobs, int32_t num_jobs, const int32_t* expert_ids, const int32_t* num_segments_dev,
                                       int32_t num_segments, int32_t num_experts, int32_t* slot_table, void* stream) {
  return page_coded_experts_impl(jobs, num_jobs, expert_ids, num_segments_dev, num_segments, num_experts, slot_table, true, static_cast<cudaStream_t>(stream));
}

int tris::page_experts_impl(const TrisPageJob* jobs, int num_jobs, const int32_t* expert_ids, const int32_t* num_segments_dev, int num_segments,
                            int num_experts, int32_t* slot_table, bool reset, cudaStream_t stream) {
  TRIS_REQUIRE(jobs && expert_ids && slot_table, TRIS_ERR_INVALID_ARG, "tris_page_experts: null pointer");
  TRIS_REQUIRE(num_jobs >= 1 && num_jobs <= TRIS_MAX_PAGE_JOBS, TRIS_ERR_INVALID_ARG,
               "tris_page_experts: %d jobs (1..%d supported)", num_jobs, TRIS_MAX_PAGE_JOBS);
  TRIS_REQUIRE(num_segments >= 0 && num_experts > 0, TRIS_ERR_INVALID_ARG, "tris_page_experts: bad sizes");
  if (num_segments == 0) return TRIS_OK;
  PageArgs args{};
  for (int j = 0; j < num_jobs; ++j) {
    TRIS_REQUIRE(jobs[j].host_src && jobs[j].dst && jobs[j].bytes_per_expert > 0 && (jobs[j].bytes_per_expert & 15) == 0,
                 TRIS_ERR_INVALID_ARG, "tris_page_experts: job %d needs pointers and a block size that is a multiple of 16", j);
    TRIS_REQUIRE(((reinterpret_cast<uintptr_t>(jobs[j].host_src) | reinterpret_cast<uintptr_t>(jobs[j].dst)) & 15) == 0,
                 TRIS_ERR_INVALID_ARG, "tris_page_experts: job %d buffers must be 16-byte aligned", j);
    args.jobs[j] = jobs[j];
    // the kernel dereferences the host buffer: translate to its device alias (same address under UVA)
    void* dev_alias = nullptr;
    TRIS_CUDA(cudaHostGetDevicePointer(&dev_alias, const_cast<void*>(jobs[j].host_src), 0));
    args.jobs[j].host_src = dev_alias;
  }
  args.num_jobs = num_jobs;
  args.expert_ids = expert_ids;
  args.num_segments_dev = num_segments_dev;
  args.num_segments = num_segments;
  args.num_experts = num_experts;
  args.slot_table = slot_table;
  // Experts that get no slot (more live segments than num_segments) must not keep a stale entry:
  // the grouped kernels treat -1 as "not paged in", store nothing and report TRIS_ERR_WORKSPACE.
  if (reset) TRIS_CUDA(cudaMemsetAsync(slot_table, 0xFF, sizeof(int32_t) * static_cast<size_t>(num_experts), stream));
  page_experts_kernel<<<kPagerCtas, kPageThreads, 0, stream>>>(args);
  return check_cuda(cudaGetLastError(), "page_experts_kernel launch");
}
extern "C" int tris_page_experts(const TrisPageJob* jobs, int32_t num_jobs, const int32_t* expert_ids,
                                 const int32_t* num_segments_dev, int32_t num_segments, int32_t num_experts,
                                 int32_t* slot_table, void* stream) {
  return page_experts_impl(jobs, num_jobs, expert_ids, num_segments_dev, num_segments, num_experts, slot_table, true, static_cast<cudaStream_t>(stream));
}
