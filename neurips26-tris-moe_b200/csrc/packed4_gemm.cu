// GEMMs that read GPTQ-style 4-bit matrices as they are stored (no fp16 copy in HBM):
//
//   * the null-space compensation of ns_mode == 2 experts, comp = (x . C2^T) . C1^T per routed
//     segment, with every expert's C2 / C1 inside one concatenated tensor
//     (run_grouped_ns_compensation_forward, qlinear_cuda.py:2024-2128; kernels
//     GroupedPacked4LinearOffset{Segment,Decode}{C2,C1}, TriSMoE_cuda_kernel.cu:1208-2144), and
//   * the shared backbone product hidden = x . shared_sv^T on the packed matrix
//     (_run_packed_4bit_linear_cuda, qlinear_cuda.py:1148-1168; Packed4LinearKernelTiledLop3[SplitK],
//     TriSMoE_cuda_kernel.cu:914-1104).
//
// Numerics: every weight is fp16((q - zero) * scale) with one rounding, bit for bit the matrix
// PackedQuantMatrix4bit.dequantize (qlinear_cuda.py:2756-2784) hands to F.linear in the reference's
// fallback; products accumulate in fp32 on the tensor cores and are rounded to fp16 once.
//
// Shape of the work: few activation rows (a decode batch, or the rows of one routed segment) against
// a matrix whose bytes dominate, so the matrix is the A operand of mma.m16n8k16 (16 outputs x 16
// inputs per instruction, 8 activation rows as the N side) and each nibble is expanded exactly once
// per pass, in registers.  Lane (g, t) takes word row 4s + t of outputs g and g + 8 of a 32-column slice s:
// 8 columns of each, A fragments of two K = 16 steps if step j's K positions are columns 8t + 4j .. + 3;
// the lane's activations of the slice are then 16 contiguous bytes.  Nibbles and activations are read
// straight from global memory (L2 / L1) and nothing is staged; four CTAs on an SM hide the latency
// better than loads four slices ahead in 125 registers (a whole block with null-space pairs, 37 tokens, called from Python, when C1
// took this kernel too: 128 against 148 us).  Staging 32 KB of nibbles and up to 128 KB of activation rows per CTA whatever the
// problem's size let one CTA fill an SM: 64 segments of 5 rows, 2048 -> 64 and 64 -> 1024, took 42 us a
// launch.  Gate and up share a launch.
// The eight warps of a CTA split the columns as far as there are slices and take further groups of 16 outputs
// otherwise; partial sums meet in shared memory.  What bounds it: latency of a handful of dependent
// round trips; launches.
#include <math.h>

#include <algorithm>

#include "common.cuh"

namespace tris {

constexpr int kP4Threads = 256;
constexpr int kP4Warps = 8;
constexpr int kP4TileN = 16;       // outputs of a warp
constexpr int kP4SliceCols = 32;
constexpr int kP4RedStride = 20;   // floats per (warp, activation row) in the reduction buffer

struct P4Args {
  P4Problem p[2];
  int num_problems;
  const int32_t* expert_ids;
  const int32_t* segment_offsets;
  const int32_t* num_segments_dev;
  const int32_t* row_gather;
  int num_segments;  // 0: no route, one matrix for all rows
  int num_experts;
  int num_rows;
  int out_mode;
  int accumulate;
  int n;       // outputs of either problem, at most
  int ksplit;  // warps that share 16 outputs: 1, 2, 4 or 8
  int rows_ready;  // route and rows are older than the kernel before: only the stores wait for it
};

// byte i of `word` holds the nibbles of input columns 2i (low) and 2i+1 (high): returns
// half2(fp16((q_lo - zero) * scale), fp16((q_hi - zero) * scale)); zc = 1024 + zero as half2
__device__ __forceinline__ uint32_t p4_dequant_pair(uint32_t word, int i, __half2 zc, __half2 sc) {
  const uint32_t b = prmt(word, 0u, 0x4440u + static_cast<uint32_t>(i));
  const uint32_t v = ((b * 4097u) & 0x000F000Fu) | 0x64006400u;  // 1024 + q, exact in fp16
  return h2_as_u32(__hmul2(__hsub2(u32_as_h2(v), zc), sc));
}

// A lane's view of 16 outputs of one matrix: the quantisation of a group of columns.
struct P4Group {
  __half2 za, zb, sa, sb;  // 1024 + zero and scale of outputs a and b
};
__device__ __forceinline__ P4Group p4_group(const int32_t* z, const __half* s, int na, int nb) {
  const uint32_t za = (static_cast<uint32_t>(__ldg(z + (na >> 3))) >> (4 * (na & 7))) & 0xFu;
  const uint32_t zb = (static_cast<uint32_t>(__ldg(z + (nb >> 3))) >> (4 * (nb & 7))) & 0xFu;
  return {__half2half2(__ushort_as_half(static_cast<unsigned short>(0x6400u + za + 1u))),
          __half2half2(__ushort_as_half(static_cast<unsigned short>(0x6400u + zb + 1u))), __half2half2(__ldg(s + na)), __half2half2(__ldg(s + nb))};
}
// Eight columns k .. k + 7 of a row of K; columns past K read as zeros.
__device__ __forceinline__ uint4 p4_row_piece(const __half* src, int k, int K, bool aligned) {
  if (k >= K) return make_uint4(0u, 0u, 0u, 0u);
  if (aligned && k + 8 <= K) return *reinterpret_cast<const uint4*>(src);
  uint32_t h[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) h[j] = k + j < K ? __half_as_ushort(src[j]) : 0u;
  return make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
}

// grid (groups of 16 * 8 / ksplit outputs, segments or 1, problems * CTAs that share a segment's rows)
template <int NT>
__global__ void __launch_bounds__(kP4Threads, NT <= 2 ? 4 : 2) packed4_gemm_kernel(const __grid_constant__ P4Args a) {
  constexpr int kRows = 8 * NT;
  extern __shared__ __align__(16) float red[];              // [warp][activation row][kP4RedStride]

  if (!a.rows_ready) pdl_wait();  // activations (and a device-built route) come from the kernels before this one
  pdl_launch_dependents();
  // A CTA without work leaves at once, but the first one waits: if none did, the launch could end before its predecessor.
  auto leave = [&] {
    if (a.rows_ready && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) pdl_wait();
  };
  int e = 0, row0 = 0, rows = a.num_rows;
  if (a.num_segments > 0) {
    const int seg = blockIdx.y;
    const int nseg = a.num_segments_dev ? min(*a.num_segments_dev, a.num_segments) : a.num_segments;
    if (seg >= nseg) return leave();
    e = a.expert_ids[seg];
    if (e < 0 || e >= a.num_experts) return leave();
    row0 = a.segment_offsets[seg];
    rows = min(a.segment_offsets[seg + 1], a.num_rows) - row0;
  }
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int og = warp / a.ksplit, ks = warp % a.ksplit;
  const int outs = (kP4Warps / a.ksplit) * kP4TileN;
  const int cta_n = blockIdx.x * outs, n0 = cta_n + og * kP4TileN;
  if (rows <= 0 || row0 < 0) return leave();
  const int np = a.num_problems;  // CTAs of their own for each
  const P4Problem& pr = a.p[blockIdx.z % np];
  const TrisPacked4View& w = pr.w;
  for (int r0 = (blockIdx.z / np) * kRows; r0 < rows; r0 += kRows * (gridDim.z / np)) {
    const int N = w.n_count ? w.n_count[e] : w.n;
    const int K = w.k_count ? w.k_count[e] : w.k;
    const int G = max(1, w.g_count ? w.g_count[e] : w.num_groups);
    if (cta_n >= N) return leave();
    const int n_off = w.n_off ? w.n_off[e] : 0;
    const int g_off = w.g_off ? w.g_off[e] : 0;
    // outputs past N repeat the last one
    const int na = min(n0 + g, N - 1), nb = min(n0 + g + 8, N - 1);
    const int32_t* qw = w.qweight + static_cast<size_t>(w.kw_off ? w.kw_off[e] : 0) * w.q_ld + n_off;
    const int32_t* qz = w.qzeros + static_cast<size_t>(g_off) * w.z_ld + (w.z_off ? w.z_off[e] : 0);
    const __half* sc = static_cast<const __half*>(w.scales) + static_cast<size_t>(g_off) * w.s_ld + n_off;
    const int kwords = (K + 7) >> 3, slices = (K + kP4SliceCols - 1) / kP4SliceCols;
    const int per = (slices + a.ksplit - 1) / a.ksplit;
    const int s_begin = n0 < N ? ks * per : 0, s_end = n0 < N ? min(slices, s_begin + per) : 0;
    const int gs = w.group_size > 0 ? w.group_size : (K + kP4SliceCols);  // a multiple of 32 where there are several groups
    float acc[NT][4];
    const __half* xr[NT];  // this lane's activation row of each tile; rows past the last repeat it
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
      const int r = row0 + min(r0 + 8 * i + g, rows - 1);
      xr[i] = pr.x + static_cast<size_t>(a.row_gather ? a.row_gather[r] : r) * pr.x_ld + 8 * t;
    }
    int grp = -1;
    P4Group q = {};
#pragma unroll 1
    for (int s = s_begin; s < s_end; ++s) {
      const int kw = 4 * s + t, k = 8 * kw;
      const bool in = kw < kwords;
      const uint32_t wa = in ? static_cast<uint32_t>(__ldg(qw + static_cast<size_t>(kw) * w.q_ld + na)) : 0u;
      const uint32_t wb = in ? static_cast<uint32_t>(__ldg(qw + static_cast<size_t>(kw) * w.q_ld + nb)) : 0u;
      uint4 xv[NT];
#pragma unroll
      for (int i = 0; i < NT; ++i) xv[i] = p4_row_piece(xr[i] + kP4SliceCols * s, k, K, pr.x_aligned);
      const int gi = min(s * kP4SliceCols / gs, G - 1);
      if (gi != grp) {
        grp = gi;
        q = p4_group(qz + static_cast<size_t>(gi) * w.z_ld, sc + static_cast<size_t>(gi) * w.s_ld, na, nb);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t a0 = p4_dequant_pair(wa, 2 * j, q.za, q.sa), a1 = p4_dequant_pair(wb, 2 * j, q.zb, q.sb);
        const uint32_t a2 = p4_dequant_pair(wa, 2 * j + 1, q.za, q.sa), a3 = p4_dequant_pair(wb, 2 * j + 1, q.zb, q.sb);
#pragma unroll
        for (int i = 0; i < NT; ++i) mma_m16n8k16(acc[i], a0, a1, a2, a3, j ? xv[i].z : xv[i].x, j ? xv[i].w : xv[i].y);
      }
    }
    // add the partial sums of the warps that share 16 outputs
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      float* base = red + (warp * kRows + 8 * i + 2 * t) * kP4RedStride;
      base[g] = acc[i][0];
      base[kP4RedStride + g] = acc[i][1];
      base[g + 8] = acc[i][2];
      base[kP4RedStride + g + 8] = acc[i][3];
    }
    if (a.rows_ready) pdl_wait();
    __syncthreads();
    for (int i = tid; i < min(kRows, rows - r0) * outs; i += kP4Threads) {
      const int r = i / outs, j = i - r * outs, n = cta_n + j;
      if (n >= N) continue;
      const float* src = red + ((j / kP4TileN) * a.ksplit * kRows + r) * kP4RedStride + j % kP4TileN;
      float sum = 0.f;
      for (int v = 0; v < a.ksplit; ++v) sum += src[v * kRows * kP4RedStride];
      const size_t row = static_cast<size_t>(row0 + r0 + r);
      const int col = out_mode_pos(n, a.out_mode);
      __half* dst = pr.out + row * pr.out_ld + col;
      __half v = __float2half_rn(sum);
      if (a.accumulate) v = __hadd(*dst, v);  // what out.add_(compensation) does in fp16
      *dst = v;
    }
    __syncthreads();
  }
}

// Products of few columns, as a rule added to what lies in the output: C1 of the null-space pairs.  A warp takes 32 outputs of one segment and
// all their columns, so nothing is exchanged between warps, and asks for weights, rows and old outputs at once: a launch is
// one round trip after the tables of the segment.  kSilu: both problems (gate, up) belong to a warp, and problem 0's output becomes silu(gate) *
// up, each rounded to fp16 where separate operators would round it; up's own output is not stored.
// grid (groups of 128 outputs, segments, 1 or problems), four warps.
constexpr int kP4AddWarps = 4, kP4AddN = 32;
template <int NT, bool kSilu>
__global__ void __launch_bounds__(32 * kP4AddWarps) packed4_add_kernel(const __grid_constant__ P4Args a) {
  pdl_wait();
  pdl_launch_dependents();
  const int seg = blockIdx.y;
  const int nseg = a.num_segments_dev ? min(*a.num_segments_dev, a.num_segments) : a.num_segments;
  if (seg >= nseg) return;
  const int e = a.expert_ids[seg];
  if (e < 0 || e >= a.num_experts) return;
  const int row0 = a.segment_offsets[seg], rows = min(a.segment_offsets[seg + 1], a.num_rows) - row0;
  if (rows <= 0 || row0 < 0) return;
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = (blockIdx.x * kP4AddWarps + warp) * kP4AddN;

  // sum of x . W^T for rows r0 .. of 32 outputs
  auto product = [&](const P4Problem& pr, int N, int r0, float (&acc)[2][NT][4]) {
    const TrisPacked4View& w = pr.w;
    const int K = w.k_count ? w.k_count[e] : w.k, G = max(1, w.g_count ? w.g_count[e] : w.num_groups);
    const int n_off = w.n_off ? w.n_off[e] : 0, g_off = w.g_off ? w.g_off[e] : 0;
    const int32_t* qw = w.qweight + static_cast<size_t>(w.kw_off ? w.kw_off[e] : 0) * w.q_ld + n_off;
    const int32_t* qz = w.qzeros + static_cast<size_t>(g_off) * w.z_ld + (w.z_off ? w.z_off[e] : 0);
    const __half* sc = static_cast<const __half*>(w.scales) + static_cast<size_t>(g_off) * w.s_ld + n_off;
    const int kwords = (K + 7) >> 3, slices = (K + kP4SliceCols - 1) / kP4SliceCols;
    const int gs = w.group_size > 0 ? w.group_size : (K + kP4SliceCols);
    const __half* xr[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int r = row0 + min(r0 + 8 * i + g, rows - 1);
      xr[i] = pr.x + static_cast<size_t>(a.row_gather ? a.row_gather[r] : r) * pr.x_ld + 8 * t;
    }
    int grp = -1;
    P4Group q[2] = {};
#pragma unroll 1
    for (int s0 = 0; s0 < slices; s0 += 2) {  // two slices in flight
      uint32_t wv[2][4];
      uint4 xv[2][NT];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int kw = 4 * (s0 + u) + t;
#pragma unroll
        for (int h = 0; h < 4; ++h)
          wv[u][h] = kw < kwords ? static_cast<uint32_t>(__ldg(qw + static_cast<size_t>(kw) * w.q_ld + min(n0 + 8 * h + g, N - 1))) : 0u;
#pragma unroll
        for (int i = 0; i < NT; ++i) xv[u][i] = p4_row_piece(xr[i] + kP4SliceCols * (s0 + u), 8 * kw, K, pr.x_aligned);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int gi = min((s0 + u) * kP4SliceCols / gs, G - 1);
        if (gi != grp) {
          grp = gi;
#pragma unroll
          for (int m = 0; m < 2; ++m)
            q[m] = p4_group(qz + static_cast<size_t>(gi) * w.z_ld, sc + static_cast<size_t>(gi) * w.s_ld, min(n0 + 16 * m + g, N - 1), min(n0 + 16 * m + 8 + g, N - 1));
        }
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint32_t a0 = p4_dequant_pair(wv[u][2 * m], 2 * j, q[m].za, q[m].sa), a1 = p4_dequant_pair(wv[u][2 * m + 1], 2 * j, q[m].zb, q[m].sb);
            const uint32_t a2 = p4_dequant_pair(wv[u][2 * m], 2 * j + 1, q[m].za, q[m].sa), a3 = p4_dequant_pair(wv[u][2 * m + 1], 2 * j + 1, q[m].zb, q[m].sb);
#pragma unroll
            for (int i = 0; i < NT; ++i) mma_m16n8k16(acc[m][i], a0, a1, a2, a3, j ? xv[u][i].z : xv[u][i].x, j ? xv[u][i].w : xv[u][i].y);
          }
      }
    }
  };
  // four outputs of a row, 8 bytes where they are aligned
  auto at = [&](const P4Problem& pr, int r, int n) { return pr.out + static_cast<size_t>(row0 + r) * pr.out_ld + n; };
  auto load4 = [&](const P4Problem& pr, int N, int r, int n) {
    uint2 v = make_uint2(0u, 0u);
    if (!a.accumulate || r >= rows || n >= N) return v;
    const __half* p = at(pr, r, n);
    if (pr.out_quads && n + 4 <= N) return *reinterpret_cast<const uint2*>(p);
    uint32_t h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = n + j < N ? __half_as_ushort(p[j]) : 0u;
    return make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
  };
  const P4Problem& first = a.p[kSilu ? 0 : blockIdx.z];
  const int N0 = first.w.n_count ? first.w.n_count[e] : first.w.n, N1 = kSilu ? (a.p[1].w.n_count ? a.p[1].w.n_count[e] : a.p[1].w.n) : 0;
  if (n0 >= max(N0, N1)) return;
  // Old outputs and the product, each four outputs of a row.  Outputs from N on of the second problem keep what lies there: the first one's may
  // be more.
  auto pass = [&](const P4Problem& pr, int N, int all, int r0, uint2 (&sum)[2][NT]) {
    uint2 old[2][NT];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int i = 0; i < NT; ++i) old[m][i] = load4(pr, all, r0 + 8 * i + g, n0 + 16 * m + 8 * (t & 1) + 2 * (t & 2));
    const bool present = pr.w.num_experts > 0 && n0 < N;
    float acc[2][NT][4] = {};
    if (present) product(pr, N, r0, acc);
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        uint2 v = outputs_of_row(h2_as_u32(__floats2half2_rn(acc[m][i][0], acc[m][i][1])), h2_as_u32(__floats2half2_rn(acc[m][i][2], acc[m][i][3])), t);
        const int left = N - (n0 + 16 * m + 8 * (t & 1) + 2 * (t & 2));
        if (kSilu && left < 4) v = make_uint2(left >= 2 ? v.x : (left == 1 ? v.x & 0xFFFFu : 0u), left == 3 ? v.y & 0xFFFFu : 0u);
        if (!a.accumulate) sum[m][i] = v;
        else sum[m][i] = !present ? old[m][i] : make_uint2(h2_as_u32(__hadd2_rn(u32_as_h2(old[m][i].x), u32_as_h2(v.x))), h2_as_u32(__hadd2_rn(u32_as_h2(old[m][i].y), u32_as_h2(v.y))));
      }
  };
#pragma unroll 1
  for (int r0 = 0; r0 < rows; r0 += 8 * NT) {
    uint2 y[2][NT];
    pass(first, N0, N0, r0, y);
    if constexpr (kSilu) {
      uint2 up[2][NT];
      pass(a.p[1], N1, max(N0, N1), r0, up);
      auto silu = [](uint32_t f, uint32_t u) {
        const float2 v = __half22float2(u32_as_h2(f));
        return h2_as_u32(__hmul2_rn(__floats2half2_rn(v.x / (1.f + expf(-v.x)), v.y / (1.f + expf(-v.y))), u32_as_h2(u)));
      };
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int i = 0; i < NT; ++i) y[m][i] = make_uint2(silu(y[m][i].x, up[m][i].x), silu(y[m][i].y, up[m][i].y));
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const int r = r0 + 8 * i + g, n = n0 + 16 * m + 8 * (t & 1) + 2 * (t & 2);
        if (r >= rows) continue;
        __half* p = at(first, r, n);
        if (first.out_quads && n + 4 <= N0) {
          *reinterpret_cast<uint2*>(p) = y[m][i];
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + j < N0) p[j] = __ushort_as_half(static_cast<unsigned short>((j & 2 ? y[m][i].y : y[m][i].x) >> (16 * (j & 1))));
        }
      }
  }
}

template <int NT, bool kSilu>
static int launch_add(const P4Args& args, cudaStream_t stream, bool pdl) {
  const dim3 grid(ceil_div(args.n, kP4AddN * kP4AddWarps), args.num_segments, kSilu ? 1 : args.num_problems);
  return check_cuda(launch_kernel(packed4_add_kernel<NT, kSilu>, grid, dim3(32 * kP4AddWarps), 0, stream, pdl, 1, args), "packed4_add_kernel launch");
}
template <bool kSilu>
static int dispatch_add(const P4Args& args, int hint, cudaStream_t stream, bool pdl) {
  if (hint <= 8) return launch_add<1, kSilu>(args, stream, pdl);
  if (hint <= 16) return launch_add<2, kSilu>(args, stream, pdl);
  return launch_add<4, kSilu>(args, stream, pdl);
}

template <int NT>
static int launch_p4(const P4Args& args, dim3 grid, cudaStream_t stream, bool pdl) {
  constexpr size_t smem = static_cast<size_t>(kP4Warps) * 8 * NT * kP4RedStride * sizeof(float);
  static_assert(smem <= 48 * 1024, "reduction buffer");
  return check_cuda(launch_kernel(packed4_gemm_kernel<NT>, grid, dim3(kP4Threads), smem, stream, pdl, 1, args), "packed4_gemm_kernel launch");
}

// One launch for one or two problems on the same rows (gate and up).  `silu`: see packed4_add_kernel; needs a route and
// two problems with `accumulate`, of which one may be absent (num_experts = 0; its `w.n` is still read).
int packed4_gemm_impl(const P4Problem* problems, int num_problems, const TrisRouteView* route, int num_rows, int out_mode,
                      bool accumulate, bool silu, cudaStream_t stream, bool pdl, bool rows_ready) {
  if (num_rows == 0) return TRIS_OK;
  P4Args args{};
  args.num_problems = num_problems;
  int hint = num_rows, k = 1;
  for (int i = 0; i < num_problems; ++i) {
    const TrisPacked4View& w = problems[i].w;
    args.p[i] = problems[i];
    args.p[i].x_aligned = ((reinterpret_cast<uintptr_t>(problems[i].x) & 15u) == 0 && problems[i].x_ld % 8 == 0) ? 1 : 0;
    args.p[i].out_quads = (reinterpret_cast<uintptr_t>(problems[i].out) & 7u) == 0 && problems[i].out_ld % 4 == 0;
    args.n = std::max(args.n, w.n);
    args.num_experts = std::max(args.num_experts, w.num_experts);
    k = std::max(k, w.num_experts > 0 ? w.k : 0);
  }
  if (route) {
    TRIS_REQUIRE(route->expert_ids && route->segment_offsets && route->num_segments >= 0, TRIS_ERR_INVALID_ARG,
                 "tris_packed4_grouped_forward: incomplete route");
    if (route->num_segments == 0) return TRIS_OK;
    args.expert_ids = route->expert_ids;
    args.segment_offsets = route->segment_offsets;
    args.num_segments_dev = route->num_segments_dev;
    args.num_segments = route->num_segments;
    args.row_gather = route->row_gather;
    if (route->max_rows_per_segment > 0) hint = std::min(hint, route->max_rows_per_segment);
    // mean + 2 sigma of a balanced router: a longer segment takes several passes
    const double mean = static_cast<double>(num_rows) / route->num_segments;
    hint = std::max(1, std::min(hint, static_cast<int>(ceil(mean + 2.0 * sqrt(mean)))));
  }
  args.num_rows = num_rows;
  args.out_mode = out_mode;
  args.accumulate = accumulate ? 1 : 0;
  args.rows_ready = pdl && rows_ready;
  const int slices = ceil_div(k, kP4SliceCols);
  // Few columns of many segments (C1 of null-space pairs): a warp per 32 outputs.  64 segments, 37 tokens, pairs of rank 32 and 64, a block
  // with them, replayed as a graph, on the kernel below / on this one 107 / 87 us, 512 tokens 350 / 208, 1 token 45.9 / 46.4.
  TRIS_REQUIRE(args.num_segments <= 65535, TRIS_ERR_UNSUPPORTED, "tris_packed4_grouped_forward: more than 65535 segments");
  if (silu) return dispatch_add<true>(args, hint, stream, pdl);
  if (route && out_mode == TRIS_OUT_F16 && slices <= 4) return dispatch_add<false>(args, hint, stream, pdl);
  // eight warps share 16 outputs where there are columns for all of them, else they take more outputs
  args.ksplit = slices >= 8 ? 8 : (slices >= 4 ? 4 : (slices >= 2 ? 2 : 1));
  dim3 grid(ceil_div(args.n, kP4TileN * kP4Warps / args.ksplit), route ? route->num_segments : 1);
  // passes of 64 rows go to CTAs of their own while that leaves four per SM
  const unsigned np = static_cast<unsigned>(num_problems);
  grid.z = np * std::max(1u, std::min(static_cast<unsigned>(ceil_div(hint, 64)), 592u / std::max(1u, grid.x * grid.y * np)));
  if (hint <= 8) return launch_p4<1>(args, grid, stream, pdl);
  if (hint <= 16) return launch_p4<2>(args, grid, stream, pdl);
  if (hint <= 32) return launch_p4<4>(args, grid, stream, pdl);
  return launch_p4<8>(args, grid, stream, pdl);
}

int validate_packed4(const TrisPacked4View* w) {
  TRIS_REQUIRE(w->qweight && w->qzeros && w->scales, TRIS_ERR_INVALID_ARG, "tris_packed4_grouped_forward: null matrix pointer");
  TRIS_REQUIRE(w->n > 0 && w->k >= 0 && w->num_groups >= 0 && w->num_experts > 0 && w->q_ld > 0 && w->z_ld > 0 && w->s_ld > 0,
               TRIS_ERR_INVALID_ARG, "tris_packed4_grouped_forward: bad sizes n=%d k=%d groups=%d", w->n, w->k, w->num_groups);
  TRIS_REQUIRE(w->group_size <= 0 || w->group_size % 32 == 0 || w->num_groups <= 1, TRIS_ERR_UNSUPPORTED,
               "tris_packed4_grouped_forward: group size %d (a multiple of 32, or a single group, is supported)", w->group_size);
  return TRIS_OK;
}
}  // namespace tris

using namespace tris;

extern "C" int tris_packed4_grouped_forward(const TrisPacked4View* w, const TrisRouteView* route, const void* x_f16,
                                            int32_t x_ld, int32_t num_rows, void* out_f16, int32_t out_ld,
                                            int32_t out_mode, int32_t accumulate, void* stream) {
  TRIS_REQUIRE(w && x_f16 && out_f16, TRIS_ERR_INVALID_ARG, "tris_packed4_grouped_forward: null pointer");
  const int st = validate_packed4(w);
  if (st != TRIS_OK) return st;
  TRIS_REQUIRE(out_mode == TRIS_OUT_F16 || out_mode == TRIS_OUT_F16_PAIR_INTERLEAVED || out_mode == TRIS_OUT_F16_LANE_ORDER,
               TRIS_ERR_INVALID_ARG, "tris_packed4_grouped_forward: out_mode %d", out_mode);
  TRIS_REQUIRE(out_mode == TRIS_OUT_F16 || w->n % 32 == 0, TRIS_ERR_INVALID_ARG,
               "tris_packed4_grouped_forward: permuted output layouts need n %% 32 == 0");
  TRIS_REQUIRE(x_ld >= w->k && out_ld >= w->n && num_rows >= 0, TRIS_ERR_INVALID_ARG,
               "tris_packed4_grouped_forward: row strides x_ld=%d out_ld=%d", x_ld, out_ld);
  const P4Problem problem{*w, static_cast<const __half*>(x_f16), static_cast<__half*>(out_f16), x_ld, out_ld, 0, 0};
  return packed4_gemm_impl(&problem, 1, route, num_rows, out_mode, accumulate != 0, false, static_cast<cudaStream_t>(stream),
                           programmatic_launch_default());
}
