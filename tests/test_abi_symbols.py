"""CPU test: the shared library loads without a GPU and exports every symbol that
include/trismoe_b200.h declares; argument validation works without touching a device."""
import ctypes as C
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "trismoe_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(tris_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported(lib):
    import trismoe_b200 as tm

    names = _declared_symbols()
    assert len(names) >= 15
    for name in names:
        assert hasattr(lib, name), f"{name} declared in the header but not exported"
    assert set(names) == set(tm._native.SIGNATURES), "ctypes table and header disagree"
    assert lib.tris_abi_version() == tm._native.ABI_VERSION == 4
    assert lib.tris_compact3_kernel_abi_version() == 2


def test_status_strings_and_host_validation(lib):
    import trismoe_b200 as tm

    assert lib.tris_status_string(0) == b"ok"
    assert b"corrupt" in lib.tris_status_string(4)
    # null pointers are rejected on the host, before any CUDA call
    st = lib.tris_grouped_forward(None, None, None, None, None)
    assert st == 1
    assert b"null" in lib.tris_last_error()
    view = tm._native.TrisProjView()
    st = lib.tris_block_gr_decode(C.byref(view), None, None)
    assert st == 1
    n = C.c_int64(0)
    st = lib.tris_block_gr_encode_host(None, 1, 1, 0, None, 0, None, None, C.byref(n))
    assert st == 1


def test_struct_sizes_match_c_layout(lib):
    """ctypes mirrors of the ABI structs: natural alignment, no packing surprises."""
    import trismoe_b200 as tm

    assert C.sizeof(tm._native.TrisProjView) == 224  # static_assert in csrc/common.cuh
    assert tm._native.TrisProjView.tile_records.offset == 184
    assert C.sizeof(tm._native.TrisRouteView) == 80
    assert C.sizeof(tm._native.TrisPacked4View) == 112
    assert tm._native.TrisRouteView.row_gather.offset == 40
    assert tm._native.TrisRouteView.out_row_scatter.offset == 64
    assert C.sizeof(tm._native.TrisSharedExpert) == 32
    assert C.sizeof(tm._native.TrisPageLaunch) == 24
    assert C.sizeof(tm._native.TrisPagedLayer) == 1472
    assert tm._native.TrisPagedLayer.staged.offset == 24 and tm._native.TrisPagedLayer.timing.offset == 1424


def test_cpu_tensors_are_rejected_loudly(lib):
    import pytest
    import torch
    import trismoe_b200 as tm

    with pytest.raises(RuntimeError, match="CUDA"):
        tm.compute_shared_hidden(torch.zeros(2, 8, dtype=torch.float16), torch.zeros(4, 8, dtype=torch.float16))
    with pytest.raises(RuntimeError, match="CUDA"):
        tm.build_grouped_route(torch.zeros(2, 2, dtype=torch.long), 4)


def _record_view(out_features, rank):
    """A projection with tile records as the host rules see it; the addresses are never followed."""
    import trismoe_b200 as tm

    v = tm._native.TrisProjView()
    v.num_experts, v.out_features, v.rank, v.num_groups, v.use_block_gr = 1, out_features, rank, 1, 1
    v.tile_records = v.col_records = 1 << 20
    v.col_record_bytes, v.max_record_bytes, v.max_sal_words = 672, 4 * 1408, 1
    return v


def test_column_split_scratch_is_bounded(lib):
    need = lambda o, rank, projections, rows: lib.tris_linear_workspace_bytes(C.byref(_record_view(o, rank)), projections, rows)
    assert need(4096, 4096, 1, 512) == 2 * 4 * 512 * 4096 and need(1024, 4096, 2, 512) == 4 * 2 * 4 * 512 * 1024
    assert need(4096, 4096, 1, 4096) == 2 * 4 * 4096 * 4096
    for o, rank, projections in ((1024, 4096, 2), (256, 8192, 1), (72, 2048, 1), (4096, 4096, 1)):
        for rows in (33, 1000, 16384, 100_000, 1 << 20, (1 << 31) - 1):
            n = need(o, rank, projections, rows)
            assert n <= 256 << 20 and n % (4 * projections * rows * o) == 0


def test_scratch_of_attention_projections_is_that_of_the_largest_launch(lib):
    one = lambda view, n, rows: lib.tris_linear_workspace_bytes(C.byref(view), n, rows)
    for widths, rank in (((4096, 1024, 1024), 4096), ((256, 1024, 1024), 2048), ((512, 256, 4096), 2048), ((2048, 128, 64), 4096)):
        q, k, v = (_record_view(w, rank) for w in widths)
        for rows in (1, 32, 33, 100, 512, 3000):
            launches = [(q, 1), (k, 2)] if widths[1] == widths[2] else [(q, 1), (k, 1), (v, 1)]
            want = max(one(view, n, rows) for view, n in launches)
            assert lib.tris_qkv_workspace_bytes(q, k, v, rows) == want and (want > 0) == (rows > 32)


def test_misaligned_workspace_of_an_ordinary_matrix_is_refused(lib):
    """The sums of the column parts are read 16 bytes at a time.  Refused before any CUDA call, so no GPU is needed."""
    import trismoe_b200 as tm

    view, route = _record_view(256, 1024), tm._native.TrisRouteView()
    route.num_segments, route.num_rows, route.max_rows_per_segment = 1, 64, 64
    need = lib.tris_linear_workspace_bytes(C.byref(view), 1, 64)
    assert need > 0
    st = lib.tris_linear_forward(C.byref(view), None, C.byref(route), 4096, None, 8192, None, 0, 16388, need, None)
    assert st == 1 and b"16-byte aligned" in lib.tris_last_error()


def test_outputs_that_the_combine_cannot_store_are_refused(lib):
    """Rows of y are stored 16 bytes at a time.  Refused before any CUDA call by every form of the layer."""
    import trismoe_b200 as tm

    def layer(H):
        v = tm._native.TrisMoeLayerView()
        v.hidden_size, v.intermediate_size, v.num_experts, v.top_k = H, 96, 1, 1
        v.gate, v.up, v.down = _record_view(96, 64), _record_view(96, 64), _record_view(H, 64)
        for name in ("router_weight", "shared_gate", "shared_up", "shared_down"):
            setattr(v, name, 1 << 20)
        return v

    def shared(H):
        views = [_record_view(32, H), _record_view(32, H), _record_view(H, 32)]
        return tm._native.TrisSharedExpert(*(C.addressof(v) for v in views), 1 << 20), views

    for H, y, status in ((64, (1 << 20) + 8, 1), (100, 1 << 20, 2)):
        view, (expert, keep) = layer(H), shared(H)
        calls = [lambda: lib.tris_moe_layer_forward(C.byref(view), 1 << 20, None, 3, y, None, 1 << 20, 1 << 30, None),
                 lambda: lib.tris_moe_layer_forward_extras(C.byref(view), C.byref(tm._native.TrisMoeLayerExtras()), 1 << 20, None, 3, y, None, 1 << 20, 1 << 30, None),
                 lambda: lib.tris_moe_layer_forward_shared(C.byref(view), C.byref(expert), 1 << 20, None, 3, y, None, 1 << 20, 1 << 30, None, 0, None)]
        for call in calls:
            assert call() == status and (b"aligned" if status == 1 else b"multiple of 8") in lib.tris_last_error()
