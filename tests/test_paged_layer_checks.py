"""CPU tests of what a streamed layer's native call refuses before it launches anything; the addresses are never followed."""
import ctypes as C

import pytest

INVALID, UNSUPPORTED = 1, 2  # TRIS_ERR_INVALID_ARG, TRIS_ERR_UNSUPPORTED
ADDRESS = 1 << 20
H, I, E, RANK = 64, 96, 8, 64


def _view(tm, out_features, rank=RANK):
    v = tm._native.TrisProjView()
    v.num_experts, v.out_features, v.rank, v.num_groups, v.gmap_sparse_rows = E, out_features, rank, 1, 2
    for name in ("qweight1", "q_gmap_sparse", "q_gmap_sparse_prefix", "c_map", "col_pack3", "row_pack3", "packed_row_group", "gmap_slot"):
        setattr(v, name, ADDRESS)
    return v


def _layer(tm, ranks=(RANK, RANK, RANK)):
    layer, paged = tm._native.TrisMoeLayerView(), tm._native.TrisPagedLayer()
    layer.hidden_size, layer.intermediate_size, layer.num_experts, layer.top_k = H, I, E, 2
    for name in ("router_weight", "shared_gate", "shared_up", "shared_down"):
        setattr(layer, name, ADDRESS)
    layer.gate, layer.up, layer.down = (_view(tm, o, r) for o, r in zip((I, I, H), ranks))
    for i, name in enumerate(("gate", "up", "down")):
        paged.staged[i] = getattr(layer, name)
    paged.slot_ids, paged.capacity, paged.copy_stream = ADDRESS, E, ADDRESS
    paged.event_route = paged.event_consumed = ADDRESS
    paged.event_paged[:] = [ADDRESS, ADDRESS]
    return layer, paged


def _with_records(paged):
    """Record views as the staging manager makes them, one salient step and one row-scale slot."""
    for i in range(3):
        r = type(paged.staged[i]).from_buffer_copy(paged.staged[i])
        r.use_block_gr, r.gmap_slot, r.tile_records, r.col_records = 1, None, ADDRESS, ADDRESS
        r.max_sal_words, r.max_record_bytes, r.col_record_bytes = 1, 4 * 1408, 672
        paged.records[i] = r
    return paged


def _call(lib, layer, paged, tokens=3):
    need = lib.tris_moe_layer_workspace_bytes(C.byref(layer), tokens)
    assert need > 0
    return lib.tris_moe_layer_forward_paged(C.byref(layer), C.byref(paged), ADDRESS, None, tokens, ADDRESS, None, ADDRESS, need, ADDRESS, None)


@pytest.mark.parametrize("records", [False, True])
@pytest.mark.parametrize("field,value", [("rank", RANK + 32), ("out_features", I + 32), ("num_experts", E + 1), ("num_groups", 2), ("use_block_gr", 1)])
def test_gate_and_up_of_different_shape_or_format_are_refused(lib, field, value, records):
    import trismoe_b200 as tm

    layer, paged = _layer(tm)
    up = paged.staged[1]
    setattr(up, field, value)
    if field == "use_block_gr":  # a complete payload of the other format
        up.q_gmap_gr_words = up.q_gmap_gr_offsets = up.q_gmap_gr_meta = up.gr_index = ADDRESS
        up.gr_substreams = 32
    if field == "rank":
        layer.up.rank = value
    if records:
        _with_records(paged)
    assert _call(lib, layer, paged) == UNSUPPORTED
    assert b"must share" in lib.tris_last_error()


@pytest.mark.parametrize("which", [0, 1, 2])
def test_staged_projections_of_another_layer_are_refused(lib, which):
    """Rows are as wide as the layer's backbones, so a staged matrix of another rank would read past them."""
    import trismoe_b200 as tm

    layer, paged = _layer(tm)
    for i in ((0, 1) if which < 2 else (2,)):
        paged.staged[i].rank = RANK + 64
    assert _call(lib, layer, paged) == INVALID and b"not the layer's" in lib.tris_last_error()


@pytest.mark.parametrize("name", ["qweight1", "c_map", "col_pack3", "row_pack3", "q_gmap_sparse_prefix"])
def test_staged_projections_with_missing_tensors_are_refused(lib, name):
    import trismoe_b200 as tm

    layer, paged = _layer(tm)
    setattr(paged.staged[2], name, None)
    assert _call(lib, layer, _with_records(paged)) == INVALID


@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("name", ["output_scale", "bias"])
@pytest.mark.parametrize("where", ["staged", "records"])
def test_records_with_a_scale_or_a_bias_are_refused(lib, which, name, where):
    """They would be read at a segment's number in place of its expert's."""
    import trismoe_b200 as tm

    layer, paged = _layer(tm)
    _with_records(paged)
    setattr(getattr(paged, where)[which], name, ADDRESS)
    assert _call(lib, layer, paged) == INVALID and b"output scale or a bias" in lib.tris_last_error()
