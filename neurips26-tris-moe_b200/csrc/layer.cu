// Whole MoE block as one stream-ordered launch sequence (no host synchronisation):
//   router logits + both input-side backbones  (one skinny-GEMM launch sharing x)
//   softmax/top-k, grouped route
//   grouped gate/up with SiLU*mul epilogue
//   down backbone on the routed rows
//   grouped down
//   weighted combine back to token order
// Input scales and null-space pairs (TrisMoeLayerExtras) join the same sequence: each matrix C2 in the wake of the grouped launch whose
// outputs its pair corrects, each C1 after it; of gate and up in one launch each, SiLU*mul in the epilogue of the second.
// A shared expert's (TrisSharedExpert) gate/up launch follows the route and its down launch the down backbone.  Both read rows that are older
// than the kernel before them and, at a few rows, wait only before they store: they run beside the route's one CTA and the down
// backbone's few.  256 experts of 512, 16 tokens, the whole layer with the two linears and the sum as operators of their own / here:
// replayed as a graph 67.5 / 47.8 us, called from Python, where the host bounds it, 119 / 51.
#include <algorithm>
#include <mutex>

#include "common.cuh"

namespace tris {
struct LayerWorkspace {
  float* logits;
  int32_t* selected;
  float* weights;
  int32_t* perm;
  int32_t* tok;
  int32_t* slot;
  int32_t* row_of_flat;
  int32_t* expert_ids;
  int32_t* segment_offsets;
  int32_t* problem_offsets;
  int32_t* counts;
  __half* hidden_gate;
  __half* hidden_up;
  __half* mlp;
  __half* hidden_down;
  __half* down_out;
  __half* up_out;       // gate/up outputs are kept apart where a null-space pair is added to either
  __half* ns_hidden[2];
  __half* scaled;
  __half* shared_mlp;   // the shared expert's rows
  __half* shared_out;
  size_t bytes;
};

static int ns_hidden_ld(const TrisPacked4View* c2) { return (c2->n + 7) & ~7; }

static LayerWorkspace carve(const TrisMoeLayerView* L, int T, char* base, const TrisMoeLayerExtras* X = nullptr,
                            const TrisSharedExpert* S = nullptr) {
  LayerWorkspace w{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* p = base ? base + off : nullptr;
    off += (bytes + 255) & ~static_cast<size_t>(255);
    return p;
  };
  const size_t R = static_cast<size_t>(T) * L->top_k;
  const size_t E = L->num_experts;
  w.counts = reinterpret_cast<int32_t*>(take(16));  // {segments, problem tiles, status, -}: first, so the status word is at a fixed offset
  w.logits = reinterpret_cast<float*>(take(sizeof(float) * T * E));
  w.selected = reinterpret_cast<int32_t*>(take(4 * R));
  w.weights = reinterpret_cast<float*>(take(4 * R));
  w.perm = reinterpret_cast<int32_t*>(take(4 * R));
  w.tok = reinterpret_cast<int32_t*>(take(4 * R));
  w.slot = reinterpret_cast<int32_t*>(take(4 * R));
  w.row_of_flat = reinterpret_cast<int32_t*>(take(4 * R));
  w.expert_ids = reinterpret_cast<int32_t*>(take(4 * E));
  w.segment_offsets = reinterpret_cast<int32_t*>(take(4 * (E + 1)));
  w.problem_offsets = reinterpret_cast<int32_t*>(take(4 * (E + 1)));
  w.hidden_gate = reinterpret_cast<__half*>(take(2 * static_cast<size_t>(T) * L->gate.rank));
  w.hidden_up = reinterpret_cast<__half*>(take(2 * static_cast<size_t>(T) * L->up.rank));
  w.mlp = reinterpret_cast<__half*>(take(2 * R * L->intermediate_size));
  w.hidden_down = reinterpret_cast<__half*>(take(2 * R * L->down.rank));
  w.down_out = reinterpret_cast<__half*>(take(2 * R * L->hidden_size));
  if (X != nullptr) {
    const bool gu = X->ns_c2[0] || X->ns_c2[1];
    w.up_out = reinterpret_cast<__half*>(take(gu ? 2 * R * L->intermediate_size : 0));
    size_t ld[2] = {0, 0};
    for (int i = 0; i < 3; ++i)
      if (X->ns_c2[i]) ld[i & 1] = std::max<size_t>(ld[i & 1], ns_hidden_ld(X->ns_c2[i]));
    for (int i = 0; i < 2; ++i) w.ns_hidden[i] = reinterpret_cast<__half*>(take(2 * R * ld[i]));
    size_t scaled = 0;
    if (X->input_scale[0] || X->input_scale[1]) scaled = static_cast<size_t>(T) * L->hidden_size;
    if (X->input_scale[2]) scaled = std::max(scaled, R * static_cast<size_t>(L->intermediate_size));
    w.scaled = reinterpret_cast<__half*>(take(2 * scaled));
  }
  if (S != nullptr) {
    w.shared_mlp = reinterpret_cast<__half*>(take(2 * static_cast<size_t>(T) * S->gate->out_features));
    w.shared_out = reinterpret_cast<__half*>(take(2 * static_cast<size_t>(T) * L->hidden_size));
  }
  w.bytes = off;
  return w;
}

// out = x * scale, rounded to fp16 (what the separate operators feed the backbone with)
__global__ void scale_columns_kernel(const __half* x, const __half* scale, size_t count, int cols, __half* out) {
  pdl_wait();
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < count; i += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[i] = __hmul(x[i], scale[i % cols]);
}

static int launch_scale_columns(const __half* x, const void* scale, int rows, int cols, __half* out, cudaStream_t s) {
  const size_t count = static_cast<size_t>(rows) * cols;
  return check_cuda(launch_kernel(scale_columns_kernel, dim3(static_cast<unsigned>(std::min<size_t>((count + 255) / 256, 1184))), dim3(256), 0, s, true, 1, x,
                                  static_cast<const __half*>(scale), count, cols, out),
                    "scale_columns_kernel launch");
}

static int validate_extras(const TrisMoeLayerView* L, const TrisMoeLayerExtras* X) {
  for (int i = 0; i < 3; ++i) {
    const TrisPacked4View *c2 = X->ns_c2[i], *c1 = X->ns_c1[i];
    TRIS_REQUIRE((c2 == nullptr) == (c1 == nullptr), TRIS_ERR_INVALID_ARG, "moe layer: null-space pair %d is incomplete", i);
    if (c2 == nullptr) continue;
    int st = validate_packed4(c2);
    if (st == TRIS_OK) st = validate_packed4(c1);
    if (st != TRIS_OK) return st;
    const int in = i == 2 ? L->intermediate_size : L->hidden_size, out = i == 2 ? L->hidden_size : L->intermediate_size;
    TRIS_REQUIRE(c2->k == in && c1->n == out && c1->k == c2->n && c2->num_experts == L->num_experts && c1->num_experts == L->num_experts,
                 TRIS_ERR_INVALID_ARG, "moe layer: null-space pair %d does not match the layer", i);
  }
  return TRIS_OK;
}

static int validate_layer(const TrisMoeLayerView* L) {
  TRIS_REQUIRE(L != nullptr, TRIS_ERR_INVALID_ARG, "moe layer: null view");
  TRIS_REQUIRE(L->hidden_size > 0 && L->intermediate_size > 0 && L->num_experts > 0 && L->top_k > 0 &&
                   L->top_k <= L->num_experts,
               TRIS_ERR_INVALID_ARG, "moe layer: bad dims H=%d I=%d E=%d k=%d", L->hidden_size, L->intermediate_size,
               L->num_experts, L->top_k);
  const bool packed_gu = L->packed_gate && L->packed_up;
  TRIS_REQUIRE((packed_gu || (L->shared_gate && L->shared_up)) && (L->packed_down || L->shared_down), TRIS_ERR_INVALID_ARG,
               "moe layer: backbone matrices missing");
  TRIS_REQUIRE(!packed_gu || (L->packed_gate->n == L->gate.rank && L->packed_up->n == L->up.rank &&
                              L->packed_gate->k == L->hidden_size && L->packed_up->k == L->hidden_size),
               TRIS_ERR_INVALID_ARG, "moe layer: packed gate/up backbones do not match rank / hidden size");
  TRIS_REQUIRE(!L->packed_down || (L->packed_down->n == L->down.rank && L->packed_down->k == L->intermediate_size),
               TRIS_ERR_INVALID_ARG, "moe layer: packed down backbone does not match rank / intermediate size");
  TRIS_REQUIRE(L->gate.out_features == L->intermediate_size && L->up.out_features == L->intermediate_size &&
                   L->down.out_features == L->hidden_size,
               TRIS_ERR_INVALID_ARG, "moe layer: projection out_features do not match H/I");
  TRIS_REQUIRE(L->gate.num_experts == L->num_experts && L->up.num_experts == L->num_experts &&
                   L->down.num_experts == L->num_experts,
               TRIS_ERR_INVALID_ARG, "moe layer: projection expert counts differ");
  return TRIS_OK;
}

static int validate_shared(const TrisMoeLayerView* L, const TrisSharedExpert* S) {
  TRIS_REQUIRE(S->gate && S->up && S->down && S->gate_weight, TRIS_ERR_INVALID_ARG, "moe layer: the shared expert is incomplete");
  TRIS_REQUIRE(S->gate->num_experts == 1 && S->up->num_experts == 1 && S->down->num_experts == 1 && S->gate->rank == L->hidden_size &&
                   S->up->rank == L->hidden_size && S->up->out_features == S->gate->out_features && S->gate->out_features > 0 &&
                   S->down->rank == S->gate->out_features && S->down->out_features == L->hidden_size,
               TRIS_ERR_INVALID_ARG, "moe layer: the shared expert does not match the layer");
  TRIS_REQUIRE(proj_has_tile_records(*S->gate) && proj_has_tile_records(*S->up) && proj_has_tile_records(*S->down), TRIS_ERR_UNSUPPORTED,
               "moe layer: the shared expert needs tile records");
  return TRIS_OK;
}

// The last kernel of a layer stores 16 bytes at a time.
static int validate_output(const TrisMoeLayerView* L, const void* y) {
  TRIS_REQUIRE((L->hidden_size & 7) == 0, TRIS_ERR_UNSUPPORTED, "moe layer: hidden_size must be a multiple of 8");
  TRIS_REQUIRE((reinterpret_cast<uintptr_t>(y) & 15u) == 0, TRIS_ERR_INVALID_ARG, "moe layer: y must be 16-byte aligned");
  return TRIS_OK;
}

// The staged projections of a streamed layer: what the grouped entry points ask of them, here before anything is launched, since the record
// kernels are launched without those entry points.
static int validate_paged(const TrisMoeLayerView* L, const TrisPagedLayer* P) {
  const TrisProjView* own[3] = {&L->gate, &L->up, &L->down};
  for (int i = 0; i < 3; ++i) {
    const int st = validate_grouped_view(P->staged + i, "tris_moe_layer_forward_paged");
    if (st != TRIS_OK) return st;
  }
  const int st = validate_pair(P->staged[0], P->staged[1]);
  if (st != TRIS_OK) return st;
  for (int i = 0; i < 3; ++i)
    TRIS_REQUIRE(P->staged[i].num_experts == own[i]->num_experts && P->staged[i].out_features == own[i]->out_features && P->staged[i].rank == own[i]->rank,
                 TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward_paged: staged projection %d is not the layer's", i);
  // a record's number is that of its segment, by which scales and biases are not indexed
  for (int i = 0; i < 3 && P->records[0].tile_records; ++i)
    TRIS_REQUIRE(!P->staged[i].output_scale && !P->staged[i].bias && !P->records[i].output_scale && !P->records[i].bias, TRIS_ERR_INVALID_ARG,
                 "tris_moe_layer_forward_paged: projection %d has an output scale or a bias, which records cannot have", i);
  return TRIS_OK;
}

// One or two 4-bit backbones on the same dense rows.
static int launch_packed(const TrisPacked4View* const* w, int count, const __half* x, int rows, int cols, __half* out0, __half* out1,
                         int out_mode, cudaStream_t s) {
  P4Problem p[2] = {};
  for (int i = 0; i < count; ++i) {
    const int st = validate_packed4(w[i]);
    if (st != TRIS_OK) return st;
    p[i] = {*w[i], x, i ? out1 : out0, cols, w[i]->n, 0};
  }
  // Overlapped where the columns are few: with 4096 and 14336 columns and 8 experts a block of 1 and 32 tokens took 74.5 and 120.6 us so, and
  // 52.7 and 113.9 with launches that wait for the one before.
  return packed4_gemm_impl(p, count, nullptr, rows, out_mode, false, false, s, /*pdl=*/cols <= 2048);
}
}  // namespace tris

using namespace tris;

extern "C" size_t tris_moe_layer_workspace_bytes(const TrisMoeLayerView* layer, int32_t num_tokens) {
  if (layer == nullptr || num_tokens < 0 || validate_layer(layer) != TRIS_OK) return 0;
  return carve(layer, num_tokens, nullptr).bytes;
}

struct SharedCall {
  const TrisSharedExpert* expert = nullptr;
  void* scratch = nullptr;
  size_t scratch_bytes = 0;
};

static int layer_forward(const TrisMoeLayerView* layer, const TrisMoeLayerExtras* extras, const void* x_f16,
                         const float* router_logits, int32_t num_tokens, void* y_f16, float* router_logits_out, void* workspace,
                         size_t workspace_bytes, int32_t* status, void* stream, const SharedCall& shared = {}) {
  int st = validate_layer(layer);
  if (st == TRIS_OK && extras) st = validate_extras(layer, extras);
  if (st == TRIS_OK && shared.expert) st = validate_shared(layer, shared.expert);
  if (st != TRIS_OK) return st;
  TRIS_REQUIRE(x_f16 && y_f16, TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward: null x/y");
  TRIS_REQUIRE(num_tokens >= 0, TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward: negative token count");
  TRIS_REQUIRE(router_logits || layer->router_weight, TRIS_ERR_INVALID_ARG,
               "tris_moe_layer_forward: need router_logits or a router weight");
  if (num_tokens == 0) return TRIS_OK;
  st = validate_output(layer, y_f16);
  if (st != TRIS_OK) return st;
  const int T = num_tokens;
  TRIS_REQUIRE(workspace != nullptr, TRIS_ERR_WORKSPACE, "tris_moe_layer_forward: null workspace");
  LayerWorkspace w = carve(layer, T, static_cast<char*>(workspace), extras, shared.expert);
  TRIS_REQUIRE(workspace_bytes >= w.bytes, TRIS_ERR_WORKSPACE, "tris_moe_layer_forward: workspace %zu < %zu bytes",
               workspace_bytes, w.bytes);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int R = T * layer->top_k;
  const __half* x = static_cast<const __half*>(x_f16);
  const void* scale_of[3] = {extras ? extras->input_scale[0] : nullptr, extras ? extras->input_scale[1] : nullptr,
                             extras ? extras->input_scale[2] : nullptr};

  // Launch order.  With logits given, router + route run first, so that the grouped
  // gate/up kernel can stage its weights while the backbone GEMM is still running
  // (programmatic dependent launch); otherwise the logits come out of the backbone GEMM.
  // Activation layout between the backbone GEMMs and the grouped kernels: row-major for the
  // tile-record kernels, pair-interleaved for the plane-staging kernels, row-major for odd ranks.
  TrisRouteView route{};
  route.num_segments = std::min(layer->num_experts, R);
  route.num_rows = R;
  route.max_rows_per_segment = T;  // top-k experts of a token are distinct
  auto hidden_mode = [&](const TrisProjView& a, const TrisProjView& b) {
    return tris_grouped_hidden_layout(&a, &b, route.num_rows, route.num_segments, route.max_rows_per_segment);
  };
  auto route_flags = [](int mode) {
    return mode == TRIS_OUT_F16_PAIR_INTERLEAVED ? TRIS_ROUTE_HIDDEN_PAIR_INTERLEAVED : 0;
  };
  const int gu_mode = hidden_mode(layer->gate, layer->up);
  const int down_mode = hidden_mode(layer->down, layer->down);
  SkinnyProblem probs[3];
  int np = 0;
  const bool packed_gu = layer->packed_gate && layer->packed_up;  // 4-bit backbones are read in place
  const SkinnyProblem gu[2] = {{static_cast<const __half*>(layer->shared_gate), w.hidden_gate, layer->gate.rank, gu_mode},
                               {static_cast<const __half*>(layer->shared_up), w.hidden_up, layer->up.rank, gu_mode}};
  for (int i = 0; i < 2; ++i)
    if (!packed_gu && !scale_of[i]) probs[np++] = gu[i];
  const bool logits_given = router_logits != nullptr;
  const float* logits = router_logits;
  if (logits_given) {
    if (router_logits_out && router_logits_out != router_logits)
      TRIS_CUDA(cudaMemcpyAsync(router_logits_out, router_logits, sizeof(float) * T * layer->num_experts,
                                cudaMemcpyDeviceToDevice, s));
  } else {
    float* dst = router_logits_out ? router_logits_out : w.logits;
    probs[np++] = {static_cast<const __half*>(layer->router_weight), dst, layer->num_experts, TRIS_OUT_F32};
    logits = dst;
  }
  auto route_launch = [&]() {
    return launch_router_route(logits, T, layer->num_experts, layer->top_k, layer->norm_topk_prob, 4, w.selected,
                               w.weights, w.perm, w.tok, w.slot, w.row_of_flat, w.expert_ids, w.segment_offsets,
                               w.problem_offsets, w.counts, s,
                               // nothing uses the grouped-down output buffer before the route exists: scratch of the
                               // multi-CTA route
                               reinterpret_cast<int32_t*>(w.down_out), 2 * static_cast<size_t>(R) * layer->hidden_size);
  };
  if (logits_given) {
    st = route_launch();
    if (st != TRIS_OK) return st;
  }
  if (np > 0) {
    // as the first launch of the sequence it may follow the kernel that wrote the matrices
    st = launch_shared_hidden(probs, np, x, nullptr, T, layer->hidden_size, s, /*pdl=*/true, nullptr, /*matrices_before_wait=*/logits_given);
    if (st != TRIS_OK) return st;
  }
  const TrisPacked4View* packed[2] = {layer->packed_gate, layer->packed_up};
  if (packed_gu && !scale_of[0] && !scale_of[1]) {
    st = launch_packed(packed, 2, x, T, layer->hidden_size, w.hidden_gate, w.hidden_up, gu_mode, s);
    if (st != TRIS_OK) return st;
  } else {
    for (int i = 0; i < 2; ++i) {  // one buffer: each backbone has read it when the next scaling starts
      if (!packed_gu && !scale_of[i]) continue;
      const __half* xi = x;
      if (scale_of[i]) {
        st = launch_scale_columns(x, scale_of[i], T, layer->hidden_size, w.scaled, s);
        if (st != TRIS_OK) return st;
        xi = w.scaled;
      }
      st = packed_gu ? launch_packed(packed + i, 1, xi, T, layer->hidden_size, i ? w.hidden_up : w.hidden_gate, nullptr, gu_mode, s)
                     : launch_shared_hidden(&gu[i], 1, xi, nullptr, T, layer->hidden_size, s, /*pdl=*/true, nullptr, true);
      if (st != TRIS_OK) return st;
    }
  }
  if (!logits_given) {
    st = route_launch();
    if (st != TRIS_OK) return st;
  }

  route.expert_ids = w.expert_ids;
  route.segment_offsets = w.segment_offsets;
  route.num_segments_dev = w.counts;
  route.status_dev = status ? status : w.counts + 2;

  TrisRouteView dense{};  // the shared expert: one segment with all tokens
  dense.num_segments = 1;
  dense.num_rows = dense.max_rows_per_segment = T;
  dense.status_dev = route.status_dev;
  // Every CTA of the kernel before either launch has waited before it lets its successor start, so what that kernel reads is final
  // and so are the rows here.
  LaunchOpts dense_opts;
  dense_opts.pdl = dense_opts.weights_before_wait = dense_opts.rows_ready = true;
  dense_opts.workspace = shared.scratch;
  dense_opts.workspace_bytes = shared.scratch ? shared.scratch_bytes : 0;
  if (shared.expert) {
    st = grouped_pair_forward_impl(shared.expert->gate, shared.expert->up, &dense, x, x, w.shared_mlp, nullptr, 1, s, dense_opts);
    if (st != TRIS_OK) return st;
  }

  // gate/up + SiLU*mul; rows read the per-token backbone outputs through tok[]
  route.row_gather = w.tok;
  route.flags = route_flags(gu_mode);
  LaunchOpts opts;
  opts.pdl = true;
  opts.weights_before_wait = logits_given;
  const bool ns_gu = extras && (extras->ns_c2[0] || extras->ns_c2[1]);
  P4Problem c2[2] = {}, c1[2] = {};
  int n2 = 0;
  if (ns_gu) {
    for (int i = 0; i < 2; ++i) {
      c1[i].w.n = layer->intermediate_size;
      c1[i].out = i ? w.up_out : w.mlp;
      c1[i].out_ld = layer->intermediate_size;
      if (!extras->ns_c2[i]) continue;
      const int ld = ns_hidden_ld(extras->ns_c2[i]);
      c2[n2++] = {*extras->ns_c2[i], x, w.ns_hidden[i], layer->hidden_size, ld, 0};
      c1[i] = {*extras->ns_c1[i], w.ns_hidden[i], c1[i].out, ld, layer->intermediate_size, 0};
    }
  }
  st = grouped_pair_forward_impl(&layer->gate, &layer->up, &route, w.hidden_gate, w.hidden_up, w.mlp, ns_gu ? w.up_out : nullptr,
                                 ns_gu ? 0 : 1, s, opts);
  if (st != TRIS_OK) return st;
  if (ns_gu) {
    // C2 reads x and the route, which are older than the kernel before it: it fills the SMs that the grouped kernel leaves (37 tokens of 64
    // experts, the block replayed as a graph: 83 us, 87 with C2 launches ahead of the grouped ones)
    st = packed4_gemm_impl(c2, n2, &route, R, TRIS_OUT_F16, false, false, s, true, /*rows_ready=*/true);
    if (st != TRIS_OK) return st;
    TrisRouteView rows = route;
    rows.row_gather = nullptr;
    st = packed4_gemm_impl(c1, 2, &rows, R, TRIS_OUT_F16, true, /*silu=*/true, s, true);
    if (st != TRIS_OK) return st;
  }

  // down backbone on routed rows
  const __half* mlp = w.mlp;
  if (scale_of[2]) {
    st = launch_scale_columns(w.mlp, scale_of[2], R, layer->intermediate_size, w.scaled, s);
    if (st != TRIS_OK) return st;
    mlp = w.scaled;
  }
  if (layer->packed_down) {
    st = launch_packed(&layer->packed_down, 1, mlp, R, layer->intermediate_size, w.hidden_down, nullptr, down_mode, s);
  } else {
    SkinnyProblem down{static_cast<const __half*>(layer->shared_down), w.hidden_down, layer->down.rank, down_mode};
    st = launch_shared_hidden(&down, 1, mlp, nullptr, R, layer->intermediate_size, s, /*pdl=*/true, nullptr, true);
  }
  if (st != TRIS_OK) return st;

  if (shared.expert) {
    st = grouped_forward_impl(shared.expert->down, &dense, w.shared_mlp, w.shared_out, s, dense_opts);
    if (st != TRIS_OK) return st;
  }

  // grouped down: the route is older than the GEMM before it, so weights stage early
  route.row_gather = nullptr;
  route.flags = route_flags(down_mode);
  opts.weights_before_wait = true;
  st = grouped_forward_impl(&layer->down, &route, w.hidden_down, w.down_out, s, opts);
  if (st != TRIS_OK) return st;
  if (extras && extras->ns_c2[2]) {
    const int ld = ns_hidden_ld(extras->ns_c2[2]);
    const P4Problem dc2{*extras->ns_c2[2], w.mlp, w.ns_hidden[0], layer->intermediate_size, ld, 0};
    const P4Problem dc1{*extras->ns_c1[2], w.ns_hidden[0], w.down_out, ld, layer->hidden_size, 0};
    st = packed4_gemm_impl(&dc2, 1, &route, R, TRIS_OUT_F16, false, false, s, true, /*rows_ready=*/true);
    if (st != TRIS_OK) return st;
    st = packed4_gemm_impl(&dc1, 1, &route, R, TRIS_OUT_F16, true, false, s, true);
    if (st != TRIS_OK) return st;
  }

  // combine
  if (shared.expert)
    return combine_shared_impl(w.down_out, w.row_of_flat, w.weights, T, layer->top_k, layer->hidden_size, x, shared.expert->gate_weight,
                               w.shared_out, y_f16, s);
  return combine_routed_impl(w.down_out, w.row_of_flat, w.weights, T, layer->top_k, layer->hidden_size, y_f16, s, true, /*indices_ready=*/true);
}

extern "C" int tris_moe_layer_forward(const TrisMoeLayerView* layer, const void* x_f16, const float* router_logits,
                                      int32_t num_tokens, void* y_f16, float* router_logits_out, void* workspace,
                                      size_t workspace_bytes, void* stream) {
  return layer_forward(layer, nullptr, x_f16, router_logits, num_tokens, y_f16, router_logits_out, workspace, workspace_bytes, nullptr, stream);
}

extern "C" size_t tris_moe_layer_extras_workspace_bytes(const TrisMoeLayerView* layer, const TrisMoeLayerExtras* extras, int32_t num_tokens) {
  if (layer == nullptr || extras == nullptr || num_tokens < 0 || validate_layer(layer) != TRIS_OK || validate_extras(layer, extras) != TRIS_OK)
    return 0;
  return carve(layer, num_tokens, nullptr, extras).bytes;
}

extern "C" int tris_moe_layer_forward_extras(const TrisMoeLayerView* layer, const TrisMoeLayerExtras* extras, const void* x_f16,
                                             const float* router_logits, int32_t num_tokens, void* y_f16, float* router_logits_out,
                                             void* workspace, size_t workspace_bytes, void* stream) {
  return layer_forward(layer, extras, x_f16, router_logits, num_tokens, y_f16, router_logits_out, workspace, workspace_bytes, nullptr, stream);
}

extern "C" int tris_moe_layer_forward_extras_status(const TrisMoeLayerView* layer, const TrisMoeLayerExtras* extras, const void* x_f16,
                                                    const float* router_logits, int32_t num_tokens, void* y_f16, float* router_logits_out,
                                                    void* workspace, size_t workspace_bytes, int32_t* status_dev, void* stream) {
  return layer_forward(layer, extras, x_f16, router_logits, num_tokens, y_f16, router_logits_out, workspace, workspace_bytes, status_dev, stream);
}

extern "C" size_t tris_moe_layer_shared_workspace_bytes(const TrisMoeLayerView* layer, const TrisSharedExpert* shared, int32_t num_tokens) {
  if (layer == nullptr || shared == nullptr || num_tokens < 0 || validate_layer(layer) != TRIS_OK || validate_shared(layer, shared) != TRIS_OK)
    return 0;
  return carve(layer, num_tokens, nullptr, nullptr, shared).bytes;
}

extern "C" int tris_moe_layer_forward_shared(const TrisMoeLayerView* layer, const TrisSharedExpert* shared, const void* x_f16,
                                             const float* router_logits, int32_t num_tokens, void* y_f16, float* router_logits_out,
                                             void* workspace, size_t workspace_bytes, void* scratch, size_t scratch_bytes, void* stream) {
  TRIS_REQUIRE(shared != nullptr, TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward_shared: null shared expert");
  TRIS_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 15u) == 0, TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward_shared: the scratch must be 16-byte aligned");
  return layer_forward(layer, nullptr, x_f16, router_logits, num_tokens, y_f16, router_logits_out, workspace, workspace_bytes, nullptr, stream,
                       {shared, scratch, scratch_bytes});
}

// ---- streaming mode ----------------------------------------------------------------------------
// Two streams: the pages cross the host link on one while the other computes what it has.  The router runs before the backbones, since the
// pages wait for its route; the backbones run beside them.  Paged experts become tile records, all but the paged bits of them while the
// pages are on their way: with those bits put in, 8 and 12 us, and the kernels for records, 11 and 15, gate/up and down of 102 experts of 512 x 256
// (twice) and 2048 x 256 take half of what the kernels for planes did (45 each, 78 beside a pager).  Two such layers with planes and seven calls
// a layer from Python / here: replayed as a graph, 16 tokens 402 / 356 us, 1 token 121 / 104; called from Python, 16 tokens 433 / 371.
extern "C" int tris_moe_layer_forward_paged(const TrisMoeLayerView* layer, const TrisPagedLayer* paged, const void* x_f16, const float* router_logits,
                                            int32_t num_tokens, void* y_f16, float* router_logits_out, void* workspace, size_t workspace_bytes,
                                            int32_t* status_dev, void* stream) {
  int st = validate_layer(layer);
  if (st != TRIS_OK) return st;
  TRIS_REQUIRE(paged && x_f16 && y_f16 && status_dev, TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward_paged: null pointer");
  TRIS_REQUIRE(num_tokens >= 0, TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward_paged: negative token count");
  TRIS_REQUIRE(router_logits || layer->router_weight, TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward_paged: need router_logits or a router weight");
  TRIS_REQUIRE(!layer->packed_gate && !layer->packed_up && !layer->packed_down, TRIS_ERR_UNSUPPORTED, "tris_moe_layer_forward_paged: fp16 backbones only");
  TRIS_REQUIRE(paged->copy_stream && paged->event_route && paged->event_paged[0] && paged->event_paged[1] && paged->event_consumed && paged->capacity > 0,
               TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward_paged: streams, events and slots are needed");
  const bool records = paged->records[0].tile_records != nullptr;
  TRIS_REQUIRE(!records || paged->slot_ids, TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward_paged: records need slot_ids");
  if (num_tokens == 0) return TRIS_OK;
  st = validate_paged(layer, paged);
  if (st == TRIS_OK) st = validate_output(layer, y_f16);
  if (st != TRIS_OK) return st;
  const int T = num_tokens, E = layer->num_experts, R = T * layer->top_k;
  LayerWorkspace w = carve(layer, T, static_cast<char*>(workspace));
  TRIS_REQUIRE(workspace != nullptr && workspace_bytes >= w.bytes, TRIS_ERR_WORKSPACE, "tris_moe_layer_forward_paged: workspace %zu < %zu bytes",
               workspace_bytes, w.bytes);
  cudaStream_t s = static_cast<cudaStream_t>(stream), copy = static_cast<cudaStream_t>(paged->copy_stream);
  const __half* x = static_cast<const __half*>(x_f16);
  auto event = [&](void* e) { return static_cast<cudaEvent_t>(e); };
  auto time = [&](int i, cudaStream_t on) { return paged->timing[i] ? cudaEventRecord(event(paged->timing[i]), on) : cudaSuccess; };

  const float* logits = router_logits;
  if (logits == nullptr) {
    float* dst = router_logits_out ? router_logits_out : w.logits;
    const SkinnyProblem router{static_cast<const __half*>(layer->router_weight), dst, E, TRIS_OUT_F32};
    st = launch_shared_hidden(&router, 1, x, nullptr, T, layer->hidden_size, s, /*pdl=*/true);
    if (st != TRIS_OK) return st;
    logits = dst;
  } else if (router_logits_out && router_logits_out != router_logits) {
    TRIS_CUDA(cudaMemcpyAsync(router_logits_out, router_logits, sizeof(float) * T * E, cudaMemcpyDeviceToDevice, s));
  }
  st = launch_router_route(logits, T, E, layer->top_k, layer->norm_topk_prob, 4, w.selected, w.weights, w.perm, w.tok, w.slot, w.row_of_flat,
                           w.expert_ids, w.segment_offsets, w.problem_offsets, w.counts, s, reinterpret_cast<int32_t*>(w.down_out),
                           2 * static_cast<size_t>(R) * layer->hidden_size);
  if (st != TRIS_OK) return st;

  TRIS_CUDA(cudaEventRecord(event(paged->event_route), s));
  TRIS_CUDA(cudaStreamWaitEvent(copy, event(paged->event_route), 0));
  if (paged->wait_consumed) TRIS_CUDA(cudaStreamWaitEvent(copy, event(paged->event_consumed), 0));
  TRIS_CUDA(time(0, copy));
  const int segments = std::min(E, R), slots = std::min(segments, paged->capacity);
  for (int g = 0; g < 2; ++g) {
    for (int i = 0; i < paged->num_pages[g]; ++i) {
      const TrisPageLaunch& p = paged->pages[g][i];
      st = p.coded ? page_coded_experts_impl(static_cast<const TrisCodedPageJob*>(p.jobs), p.num_jobs, w.expert_ids, w.counts, slots, E, p.slot_table, !records, copy)
                   : page_experts_impl(static_cast<const TrisPageJob*>(p.jobs), p.num_jobs, w.expert_ids, w.counts, slots, E, p.slot_table, !records, copy);
      if (st != TRIS_OK) return st;
    }
    if (g == 1) TRIS_CUDA(time(1, copy));
    TRIS_CUDA(cudaEventRecord(event(paged->event_paged[g]), copy));
  }

  TrisRouteView route{};
  route.expert_ids = w.expert_ids;
  route.segment_offsets = w.segment_offsets;
  route.num_segments_dev = w.counts;
  route.num_segments = segments;
  route.num_rows = R;
  route.max_rows_per_segment = T;
  route.status_dev = status_dev;
  const TrisProjView* views = records ? paged->records : paged->staged;
  const int gu_mode = tris_grouped_hidden_layout(views, views + 1, R, segments, T), down_mode = tris_grouped_hidden_layout(views + 2, nullptr, R, segments, T);
  const SkinnyProblem gu[2] = {{static_cast<const __half*>(layer->shared_gate), w.hidden_gate, layer->gate.rank, gu_mode},
                               {static_cast<const __half*>(layer->shared_up), w.hidden_up, layer->up.rank, gu_mode}};
  st = launch_shared_hidden(gu, 2, x, nullptr, T, layer->hidden_size, s, /*pdl=*/true, nullptr, /*matrices_before_wait=*/true);
  if (st != TRIS_OK) return st;
  // Records are those of the segments, in their order: place s holds segment s.
  auto paged_route = [&](int g) {
    TrisRouteView r = route;
    if (records) r.expert_ids = paged->slot_ids;
    r.row_gather = g == 0 ? w.tok : nullptr;
    r.flags = (g == 0 ? gu_mode : down_mode) == TRIS_OUT_F16_PAIR_INTERLEAVED ? TRIS_ROUTE_HIDDEN_PAIR_INTERLEAVED : 0;
    return r;
  };
  LaunchOpts opts;
  opts.pdl = records;  // after the builder; a launch that follows a wait for an event is an ordinary one
  auto arrived = [&](int g) -> int {
    TRIS_CUDA(time(2 + 2 * g, s));
    TRIS_CUDA(cudaStreamWaitEvent(s, event(paged->event_paged[g]), 0));
    TRIS_CUDA(time(3 + 2 * g, s));
    return records ? build_paged_records(paged->staged + 2 * g, paged->records + 2 * g, g == 0 ? 2 : 1, &route, paged->capacity, true, s) : static_cast<int>(TRIS_OK);
  };
  auto ahead = [&](int g) -> int {  // records as far as they do not depend on the pages
    return records ? build_paged_records(paged->staged + 2 * g, paged->records + 2 * g, g == 0 ? 2 : 1, &route, paged->capacity, false, s) : static_cast<int>(TRIS_OK);
  };
  // The builder writes the records of the ring's place, which a layer on another stream may still read.
  if (records && paged->wait_consumed) TRIS_CUDA(cudaStreamWaitEvent(s, event(paged->event_consumed), 0));
  st = ahead(0);
  if (st == TRIS_OK) st = arrived(0);
  if (st != TRIS_OK) return st;
  const TrisRouteView gu_route = paged_route(0), down_route = paged_route(1);
  st = records ? launch_grouped_tiled(views, views + 1, &gu_route, w.hidden_gate, w.hidden_up, w.mlp, nullptr, 2, route_rows_hint(&gu_route), s, opts)
               : grouped_pair_forward_impl(views, views + 1, &gu_route, w.hidden_gate, w.hidden_up, w.mlp, nullptr, 1, s, opts);
  if (st != TRIS_OK) return st;
  const SkinnyProblem down{static_cast<const __half*>(layer->shared_down), w.hidden_down, layer->down.rank, down_mode};
  st = launch_shared_hidden(&down, 1, w.mlp, nullptr, R, layer->intermediate_size, s, /*pdl=*/true, nullptr, true);
  if (st != TRIS_OK) return st;
  st = ahead(1);
  if (st == TRIS_OK) st = arrived(1);
  if (st != TRIS_OK) return st;
  st = records ? launch_grouped_tiled(views + 2, nullptr, &down_route, w.hidden_down, nullptr, w.down_out, nullptr, 0, route_rows_hint(&down_route), s, opts)
               : grouped_forward_impl(views + 2, &down_route, w.hidden_down, w.down_out, s, opts);
  if (st != TRIS_OK) return st;
  st = combine_routed_impl(w.down_out, w.row_of_flat, w.weights, T, layer->top_k, layer->hidden_size, y_f16, s, true, /*indices_ready=*/true);
  if (st != TRIS_OK) return st;
  TRIS_CUDA(cudaEventRecord(event(paged->event_consumed), s));
  return TRIS_OK;
}

// ---- variant that allocates nothing ----------------------------------------------------------
// Scratch for tris_moe_layer_forward_static.  Lives in every process image that loads the
// library, once per GPU that touches it, until the process exits.
static __device__ __align__(256) unsigned char g_layer_static_scratch[TRIS_STATIC_SCRATCH_BYTES];

namespace {
std::mutex g_static_scratch_mutex;
void* g_static_scratch_ptr[64] = {};  // device address of the array, per device ordinal
}  // namespace

extern "C" int tris_moe_layer_forward_static(const TrisMoeLayerView* layer, const void* x_f16,
                                             const float* router_logits, int32_t num_tokens, void* y_f16,
                                             float* router_logits_out, void* stream) {
  int st = validate_layer(layer);
  if (st != TRIS_OK) return st;
  TRIS_REQUIRE(num_tokens >= 0, TRIS_ERR_INVALID_ARG, "tris_moe_layer_forward_static: negative token count");
  if (num_tokens == 0) return TRIS_OK;
  LayerWorkspace probe = carve(layer, num_tokens, nullptr);
  TRIS_REQUIRE(probe.bytes <= TRIS_STATIC_SCRATCH_BYTES, TRIS_ERR_WORKSPACE,
               "tris_moe_layer_forward_static: %d tokens need %zu bytes of scratch, the built-in array holds %u; "
               "use tris_moe_layer_forward with a caller workspace",
               num_tokens, probe.bytes, static_cast<unsigned>(TRIS_STATIC_SCRATCH_BYTES));
  int dev = -1;
  TRIS_CUDA(cudaGetDevice(&dev));
  TRIS_REQUIRE(dev >= 0 && dev < 64, TRIS_ERR_UNSUPPORTED, "tris_moe_layer_forward_static: device ordinal %d", dev);
  void* scratch = nullptr;
  {
    // In host code the array's name is only a handle; the kernels need its device address,
    // which is looked up once per device with that device current.
    std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
    if (g_static_scratch_ptr[dev] == nullptr) {
      void* ptr = nullptr;
      TRIS_CUDA(cudaGetSymbolAddress(&ptr, g_layer_static_scratch));
      TRIS_REQUIRE(ptr != nullptr, TRIS_ERR_CUDA, "tris_moe_layer_forward_static: no device address for the scratch array");
      g_static_scratch_ptr[dev] = ptr;
    }
    scratch = g_static_scratch_ptr[dev];
  }
  // The array keeps whatever the previous call left.  Everything the launch sequence reads it
  // writes first, except the two count words, which are cleared here; the status word behind
  // them is sticky (it starts at zero with the array and only tris_moe_layer_last_status clears it).
  LayerWorkspace w = carve(layer, num_tokens, static_cast<char*>(scratch));
  TRIS_CUDA(cudaMemsetAsync(w.counts, 0, 8, static_cast<cudaStream_t>(stream)));
  return tris_moe_layer_forward(layer, x_f16, router_logits, num_tokens, y_f16, router_logits_out, scratch,
                                TRIS_STATIC_SCRATCH_BYTES, stream);
}

// Offset of the sticky status word inside a layer workspace (and inside the built-in scratch array).
static constexpr size_t kStatusWordOffset = 8;

extern "C" int tris_moe_layer_last_status(void* workspace, int32_t clear, void* stream, int32_t* status_out) {
  TRIS_REQUIRE(status_out != nullptr, TRIS_ERR_INVALID_ARG, "tris_moe_layer_last_status: null output");
  char* base = static_cast<char*>(workspace);
  if (base == nullptr) {  // the built-in scratch of tris_moe_layer_forward_static on the current device
    int dev = -1;
    TRIS_CUDA(cudaGetDevice(&dev));
    TRIS_REQUIRE(dev >= 0 && dev < 64, TRIS_ERR_UNSUPPORTED, "tris_moe_layer_last_status: device ordinal %d", dev);
    std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
    if (g_static_scratch_ptr[dev] == nullptr) {  // never used on this device: nothing can have been reported
      *status_out = TRIS_OK;
      return TRIS_OK;
    }
    base = static_cast<char*>(g_static_scratch_ptr[dev]);
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int32_t word = 0;
  TRIS_CUDA(cudaMemcpyAsync(&word, base + kStatusWordOffset, sizeof(word), cudaMemcpyDeviceToHost, s));
  TRIS_CUDA(cudaStreamSynchronize(s));
  if (clear && word != 0) TRIS_CUDA(cudaMemsetAsync(base + kStatusWordOffset, 0, sizeof(word), s));
  *status_out = word;
  return TRIS_OK;
}
