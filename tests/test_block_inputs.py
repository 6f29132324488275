"""CPU tests: what the MoE blocks refuse before any kernel gets an address.  The device check is taken out, so a
call that passes the checks fails later for want of a GPU, with another message."""
import pytest
import torch


@pytest.fixture
def block(monkeypatch):
    import trismoe_b200 as tm

    monkeypatch.setattr(tm._native, "require_cuda", lambda tensor, what: None)
    blk = tm.TrisSparseMoeBlock(64, 32, 4, 2)
    blk.shared_gate, blk.shared_up, blk.shared_down = (torch.zeros((32, w), dtype=torch.float16) for w in (64, 64, 32))
    return blk


@pytest.mark.parametrize("width,dtype", [(64, torch.bfloat16), (64, torch.float32), (56, torch.float16), (72, torch.float16)])
@pytest.mark.parametrize("given", [False, True])
def test_streaming_refuses_rows_it_would_misread(block, width, dtype, given):
    x = torch.zeros((1, 3, width), dtype=dtype)
    with pytest.raises(RuntimeError, match="float16 hidden states of width 64 required"):
        block.forward_streaming(x, None, 0, torch.zeros((3, 4)) if given else None)


def _calls(block, monkeypatch):
    """Which way a call took: the operators are replaced by a marker, the native sequence needs a GPU."""
    monkeypatch.setattr(block, "forward_grouped_ops", lambda x, logits=None: "operators")
    x = torch.zeros((1, 3, 64), dtype=torch.float16)
    try:
        return block(x, torch.zeros((3, 4)))
    except RuntimeError:
        return "native"


@pytest.mark.parametrize("name,count,way", [("gate", 64, "native"), ("up", 1, "operators"), ("up", 63, "operators"), ("down", 32, "native"),
                                            ("down", 64, "operators"), ("gate", 32, "operators")])
def test_input_scales_of_another_size_go_operator_by_operator(block, monkeypatch, name, count, way):
    block.input_scales = {name: torch.ones((count,), dtype=torch.float16)}
    assert _calls(block, monkeypatch) == way


@pytest.mark.parametrize("inf,outf,experts,way", [(64, 32, 4, "native"), (56, 32, 4, "operators"), (64, 40, 4, "operators"), (64, 32, 3, "operators")])
def test_null_space_pairs_of_another_size_go_operator_by_operator(block, monkeypatch, inf, outf, experts, way):
    import trismoe_b200 as tm

    c2, c1 = tm._native.TrisPacked4View(), tm._native.TrisPacked4View()
    c2.k, c1.n, c2.num_experts, c1.num_experts = inf, outf, experts, experts
    block.ns_payloads = {"up": {"_tris_ns_prepared": "cpu", "_tris_c2_view": c2, "_tris_c1_view": c1}}
    assert _calls(block, monkeypatch) == way


def test_forward_refuses_narrow_rows(block):
    with pytest.raises(RuntimeError, match="float16 hidden states of width 64 required"):
        block(torch.zeros((1, 3, 56), dtype=torch.float16), torch.zeros((3, 4)))


@pytest.mark.parametrize("gate,kernel", [(torch.zeros((1, 64)).half(), True), (torch.zeros((1, 56)).half(), False), (torch.zeros((1, 64)), False),
                                         (torch.zeros((1, 64), dtype=torch.float16, device="meta"), False)])
def test_shared_expert_gate_of_another_size_or_place(monkeypatch, gate, kernel):
    """The routed and shared outputs are replaced by tensors on the CPU: a gate that the kernel cannot take must reach
    torch's linear and its checks; one that it can take reaches the kernel (and fails for want of a GPU)."""
    import trismoe_b200 as tm
    from trismoe_b200 import compact3_linear

    blk = tm.TrisQwen2SparseMoeBlock(64, 32, 4, 2)
    x = torch.zeros((1, 3, 64), dtype=torch.float16)
    monkeypatch.setattr(tm.TrisSparseMoeBlock, "forward", lambda self, h, r=None: (torch.zeros_like(h), None))
    monkeypatch.setattr(compact3_linear, "run_compact3_gate_up_forward", lambda *a, **k: x)
    blk.shared_expert = (None, None, lambda m: torch.zeros_like(x))
    blk.shared_expert_gate.weight = torch.nn.Parameter(gate, requires_grad=False)
    linears = []
    linear = torch.nn.functional.linear
    monkeypatch.setattr(torch.nn.functional, "linear", lambda *a: linears.append(a) or linear(*a))
    try:
        blk(x)
    except (RuntimeError, ValueError):
        pass
    assert len(linears) == (0 if kernel else 1)


def test_shared_expert_gate_keeps_its_gradient(monkeypatch):
    import trismoe_b200 as tm
    from trismoe_b200 import compact3_linear

    blk = tm.TrisQwen2SparseMoeBlock(64, 32, 4, 2)
    g = torch.Generator().manual_seed(0)
    x, shared = (torch.randn((1, 3, 64), generator=g).half() for _ in range(2))
    monkeypatch.setattr(tm.TrisSparseMoeBlock, "forward", lambda self, h, r=None: (torch.zeros_like(h), None))
    monkeypatch.setattr(compact3_linear, "run_compact3_gate_up_forward", lambda *a, **k: x)
    blk.shared_expert = (None, None, lambda m: shared)
    blk.shared_expert_gate.weight = torch.nn.Parameter(torch.randn((1, 64), generator=g).half())
    y, _ = blk(x)
    y.float().sum().backward()
    z = torch.nn.functional.linear(x, blk.shared_expert_gate.weight.detach()).float()
    want = (torch.sigmoid(z) * (1 - torch.sigmoid(z)) * shared.float().sum(-1, keepdim=True) * x.float()).sum((0, 1))
    assert torch.allclose(blk.shared_expert_gate.weight.grad.float().view(-1), want, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("first,second,arrays", [(True, True, False), (True, False, True), (False, True, True), (False, False, True)])
def test_pair_of_which_one_has_no_records_gets_route_arrays(monkeypatch, first, second, arrays):
    """Only the tile-record kernels take a route without arrays, and a pair runs on them only if both have records."""
    from trismoe_b200 import compact3_linear as c3

    def linear(records):
        m = c3.Compact3Linear.__new__(c3.Compact3Linear)
        torch.nn.Module.__init__(m)
        m.payload = {"_tris_tile_records": torch.zeros(16, dtype=torch.uint8)} if records else {}
        m.in_features, m.out_features, m.input_scale = 64, 32, None
        return m

    routes = []
    monkeypatch.setattr(c3._native, "require_cuda", lambda tensor, what: None)
    monkeypatch.setattr(c3, "run_grouped_structured_expert_forward", lambda p, x, _, route: x[:, :32])
    monkeypatch.setattr(c3, "run_grouped_structured_expert_pair_forward",
                        lambda a, b, x, y, _, route, **k: routes.append(route) or (x[:, :32], y[:, :32]))
    x, a, b = torch.zeros((3, 64), dtype=torch.float16), linear(first), linear(second)
    c3.run_compact3_qkv_forward(linear(True), a, b, x)
    c3.run_compact3_gate_up_forward(a, b, x)
    assert [("expert_ids" in r, r.get("_one_segment", False)) for r in routes] == [(arrays, not arrays)] * 2


@pytest.mark.parametrize("packed,tokens", [(False, 3), (True, 3), (True, 200)])
def test_blocks_with_input_scales_share_no_scratch_between_calls(block, monkeypatch, packed, tokens):
    """Two calls in flight at once (two threads, two streams), played by a second call from inside the first one's launch:
    their workspaces and expanded backbones must not overlap.  The library is a recorder, so this needs no GPU."""
    import contextlib
    import ctypes as C
    import types

    import trismoe_b200 as tm

    spans, depth = [], []

    def forward(view, extras, x, logits, T, y, out, ws, size, *rest):
        view = view._obj
        mine = [(ws, ws + size)]
        if packed and tokens > block.PACKED_BACKBONE_MAX_ROWS:
            mine += [(getattr(view, "shared_" + n), getattr(view, "shared_" + n) + 64 * 32) for n in ("gate", "up", "down")]
        depth.append(0)
        if len(depth) == 1:
            block(torch.zeros((1, tokens, 64), dtype=torch.float16), torch.zeros((tokens, 4)))
        spans.append(mine)
        return 0

    lib = types.SimpleNamespace(tris_moe_layer_forward_extras=forward, tris_moe_layer_forward_extras_status=forward,
                                tris_moe_layer_extras_workspace_bytes=lambda *a: 4096, tris_packed4_dequantize=lambda *a: 0)
    monkeypatch.setattr(tm._native, "load", lambda: lib)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: types.SimpleNamespace(cuda_stream=0))
    view = tm._native.TrisMoeLayerView()
    block._layer_view = view
    monkeypatch.setattr(block, "layer_view", lambda: view)
    block.input_scales = {"gate": torch.ones((64,), dtype=torch.float16)}
    if packed:
        word = torch.zeros((1,), dtype=torch.int32)
        for n, w in (("gate", 64), ("up", 64), ("down", 32)):
            block.packed_backbones[n] = types.SimpleNamespace(rows=32, cols=w, groups=1, group_size=w, qweight=word, qzeros=word, scales=word)
    block(torch.zeros((1, tokens, 64), dtype=torch.float16), torch.zeros((tokens, 4)))
    assert len(spans) == 2
    for a in spans[0]:
        for b in spans[1]:
            assert a[1] <= b[0] or b[1] <= a[0]


@pytest.mark.parametrize("meta,adopted", [((672, 4 * 1408, 1), True), ((672, 4 * 2176, 1), True), ((576, 4 * 1280, 0), True), ((672, 4 * 1408, 2), False), ((768, 4 * 1408, 1), False),
                                          ((672, 4 * 1408 + 2, 1), False), ((672, 4 * 1152, 1), False), ((672, 4 * 2432, 1), False), ((0, 4 * 1408, 1), False),
                                          ((576 + 9 * 96, 4 * (1024 + 9 * 128 + 256), 9), False)])
def test_stored_records_whose_sizes_disagree_are_rebuilt(meta, adopted):
    """A checkpoint's stored tile records: the kernels compute every address from these three sizes."""
    from trismoe_b200 import qlinear_grouped as qg

    E, pr, O, rank, count = 2, 4, 100, 128, 2
    col = torch.zeros((E * meta[0],), dtype=torch.uint8)
    col[:4] = torch.tensor([qg.TILE_RECORD_MAGIC], dtype=torch.int32).view(torch.uint8)[: col.numel()]
    payload = {"_tris_gr_index": torch.zeros((E, 4, 32), dtype=torch.int32), "_tris_packed_row_group": torch.zeros((E, pr), dtype=torch.int32),
               "_tris_tile_records": torch.zeros((count * meta[1],), dtype=torch.uint8), "_tris_tile_desc": torch.zeros((count + 1, 2), dtype=torch.int32),
               "_tris_col_records": col, "_tris_tile_meta": meta, "_tris_derived_from_checkpoint": True}
    assert qg._adopt_stored_derived(payload, torch.device("cpu"), E, pr, O, rank, 1) is adopted
    assert ("_tris_tile_records" in payload) is adopted
