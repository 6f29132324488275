"""Coded pages: every bit of a bitmap comes back, at block edges, at all densities and without code where that is larger."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _code(lib, bits, per):
    E, blocks = bits.shape[0], -(-per // 1024)
    units = torch.empty((E * blocks,), dtype=torch.int32, device="cuda")
    assert lib.tris_page_code_blocks(bits.data_ptr(), per, E, units.data_ptr(), None, None, None) == 0
    offsets = torch.nn.functional.pad(units.cumsum(0, dtype=torch.int32), (1, 0)).to(torch.int32).contiguous()
    code = torch.empty((max(1, int(offsets[-1])) * 16,), dtype=torch.uint8, device="cuda")
    assert lib.tris_page_code_blocks(bits.data_ptr(), per, E, None, offsets.data_ptr(), code.data_ptr(), None) == 0
    host = torch.empty(code.shape, dtype=torch.uint8, pin_memory=True)
    host.copy_(code)
    return host, offsets, units.view(E, blocks)


@pytest.mark.parametrize("per", [16, 1008, 1024, 1040, 9 * 1024 + 528])
def test_every_bit_comes_back(lib, per):
    import trismoe_b200 as tm

    E, slots = 9, 5
    g = torch.Generator(device="cuda").manual_seed(per)
    density = torch.tensor([0.0, 1.0, 0.1, 0.02, 0.3, 0.5, 0.001, 0.1, 0.9], device="cuda")
    dense = torch.rand((E, per, 8), generator=g, device="cuda") < density.view(E, 1, 1)
    dense[7] = False
    dense[7, 0, 0] = dense[7, -1, 7] = True  # the first and the last bit
    bits = (dense.to(torch.int32) << torch.arange(8, device="cuda")).sum(2).to(torch.uint8)
    host, offsets, units = _code(lib, bits, per)
    assert (units[0] == 0).all() and (units[1, : per // 1024] == 64).all()  # nothing; left as it is
    if per >= 1024:
        assert 30 <= units[2].float()[: per // 1024].mean() <= 36  # half the size at one bit in ten
    ids = torch.tensor([8, 2, -1, 0, 7, 1, 4, 3, 5, 6], dtype=torch.int32, device="cuda")  # more experts than slots
    count = torch.tensor([ids.numel()], dtype=torch.int32, device="cuda")
    dst = torch.full((slots, per), 0xAA, dtype=torch.uint8, device="cuda")
    table = torch.zeros((E,), dtype=torch.int32, device="cuda")
    jobs = (tm._native.TrisCodedPageJob * 1)()
    jobs[0].host_src, jobs[0].block_offsets, jobs[0].dst, jobs[0].bytes_per_expert = host.data_ptr(), offsets.data_ptr(), dst.data_ptr(), per
    assert lib.tris_page_coded_experts(jobs, 1, ids.data_ptr(), count.data_ptr(), slots, E, table.data_ptr(), None) == 0
    torch.cuda.synchronize()
    want_table = [-1] * E
    for s, e in enumerate(ids.tolist()[:slots]):
        if e >= 0:
            want_table[e] = s
            assert torch.equal(dst[s], bits[e]), (s, e)
        else:
            assert (dst[s] == 0xAA).all()
    assert table.tolist() == want_table
    # an expert in every slot in turn, so that each is decoded
    for lo in range(0, E, slots):
        part = torch.arange(lo, min(E, lo + slots), dtype=torch.int32, device="cuda")
        assert lib.tris_page_coded_experts(jobs, 1, part.data_ptr(), None, part.numel(), E, table.data_ptr(), None) == 0
        torch.cuda.synchronize()
        assert torch.equal(dst[: part.numel()], bits[part.long()])
    pageable = torch.empty((bits.numel() + 64,), dtype=torch.uint8)
    assert lib.tris_page_code_blocks(bits.data_ptr(), per, E, None, offsets.data_ptr(), pageable.data_ptr(), None) == 1
    bad = (tm._native.TrisCodedPageJob * 1)()
    assert lib.tris_page_coded_experts(bad, 1, ids.data_ptr(), None, 1, E, table.data_ptr(), None) == 1
    assert lib.tris_page_coded_experts(C.cast(None, C.c_void_p), 1, ids.data_ptr(), None, 1, E, table.data_ptr(), None) == 1


def test_entry_is_coded_without_a_device_copy(lib):
    """Streaming is for GPUs whose memory is short: coding 16 MB asks for less than a thirty-second of it beside the bitmap.  Link
    bytes are those of the code, expert by expert."""
    import trismoe_b200 as tm
    from trismoe_b200 import staging

    E, rows, O = 32, 32, 4096
    g = torch.Generator(device="cuda").manual_seed(3)
    density = torch.linspace(0.0, 0.2, E, device="cuda").view(E, 1, 1)
    bitmap = torch.zeros((E, rows, O), dtype=torch.int32, device="cuda")
    for j in range(32):
        bitmap |= (torch.rand((E, rows, O), generator=g, device="cuda") < density).to(torch.int32) << j
    payload = {"qweight1": torch.zeros((E, 1, 1), dtype=torch.int32, device="cuda"), "q_gmap_sparse": bitmap}
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    entry = staging._Entry(payload, staging.BITMAP_KEYS)
    assert torch.cuda.max_memory_allocated() - before <= bitmap.numel() * 4 // 32
    per, blocks = rows * O * 4, rows * O // 256
    ends = entry.coded["q_gmap_sparse"][::blocks].tolist()
    assert entry.link_bytes["q_gmap_sparse"] == [16 * (b - a) for a, b in zip(ends, ends[1:])] and entry.link_bytes["q_gmap_sparse"][0] == 0
    assert entry.block_bytes["q_gmap_sparse"] == per and entry.rows["q_gmap_sparse"] == rows
    dst, table = torch.empty_like(bitmap), torch.empty((E,), dtype=torch.int32, device="cuda")
    jobs = (tm._native.TrisCodedPageJob * 1)()
    jobs[0].host_src, jobs[0].block_offsets = entry.host["q_gmap_sparse"].data_ptr(), entry.coded["q_gmap_sparse"].data_ptr()
    jobs[0].dst, jobs[0].bytes_per_expert = dst.data_ptr(), per
    ids = torch.arange(E, dtype=torch.int32, device="cuda")
    assert lib.tris_page_coded_experts(jobs, 1, ids.data_ptr(), None, E, E, table.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(dst, bitmap)


def test_emptied_bitmap_of_a_payload_keeps_its_type(lib):
    import trismoe_b200 as tm
    from trismoe_b200 import staging, synth

    shape = synth.LayerShape(256, 192, 8, 2, rank=96, group_size=32)
    layer = synth.synth_layer(shape, seed=6, keep_sparse_gmap=True)
    blk = tm.TrisSparseMoeBlock(256, 192, 8, 2, True)
    for name in ("gate", "up", "down"):
        layer[name]["compact3_use_block_gr"] = False
    blk.load_grouped_payloads(layer["gate"], layer["up"], layer["down"], layer["shared_gate"], layer["shared_up"], layer["shared_down"],
                              layer["router_weight"], device="cuda")
    manager = staging.GroupedQGmapCPUStagingManager([blk])
    assert manager.initialize()
    for name in ("gate", "up", "down"):
        assert manager.entries[(0, name)].coded and blk._get_grouped_payload(name)["q_gmap_sparse"].dtype == torch.int32


RECORD_SHAPES = [(256, 192, 8, 2, 96, 32, 0.1), (264, 136, 12, 3, 300, 128, 0.1), (520, 200, 6, 2, 256, 64, 0.5), (128, 72, 5, 2, 44, 32, 0.97),
                 (128, 136, 4, 2, 136, 32, 0.0)]


@pytest.mark.parametrize("H,I,E,k,rank,group,salient", RECORD_SHAPES)
@pytest.mark.parametrize("mode,sparse", [("bitmap", True), ("payload", True), ("payload", False)])
def test_paged_experts_become_the_resident_records(lib, H, I, E, k, rank, group, salient, mode, sparse):
    """Tile records built from paged planes are those of the resident block byte for byte, so that the kernels that read them give the same
    bits; salient columns from none to nearly all, one to four row-scale slots a chunk, ragged outputs and columns, one to many row tiles."""
    import numpy as np

    import trismoe_b200 as tm
    from trismoe_b200 import staging, synth

    rng = np.random.default_rng(H + rank)
    raws = {n: synth.raw_projection(rng, E, O, rank, group_size=group, p_salient=salient, col_scale_one=False)
            for n, O in (("gate", I), ("up", I), ("down", H))}
    backbones = [torch.from_numpy(rng.normal(0, 0.1, (rank, w)).astype(np.float16)) for w in (H, H, I)]
    router = torch.from_numpy(rng.standard_normal((E, H)).astype(np.float16))

    def block(sparse):
        blk = tm.TrisSparseMoeBlock(H, I, E, k, True)
        payloads = [synth.pack_projection(raws[n], "cpu", True, True) for n in ("gate", "up", "down")]
        for p in payloads:
            p["compact3_use_block_gr"] = not sparse
        return blk.load_grouped_payloads(*payloads, *backbones, router, device="cuda")

    resident, streamed = block(False), block(sparse)
    down = resident._get_grouped_payload("down")
    records, cols = down["_tris_tile_records"].view(E, -1).clone(), down["_tris_col_records"].view(E, -1).clone()
    manager = staging.GroupedQGmapCPUStagingManager([streamed], mode=mode)
    manager.initialize()
    for i, T in enumerate((1, 9, 40, 300)):
        x = synth.synth_activations(T, H, seed=T).cuda().view(1, T, H)
        logits = synth.synth_router_logits(T, E, seed=T).cuda()
        want, _ = resident(x, router_logits=logits)
        manager.collect_timings = bool(i % 2)
        got, _ = streamed.forward_streaming(x, manager, 0, router_logits=logits)
        torch.cuda.synchronize()
        assert torch.equal(got, want), T
        assert streamed.last_kernel_status() == 0
        active = sorted(set(torch.topk(torch.softmax(logits, 1), k, -1)[1].reshape(-1).tolist()))
        per, size, steps, columns = manager._record_info[(0, "down")]
        assert (per, columns) == (records.shape[1], cols.shape[1])
        buffer = manager.buffers[((manager._next - 1) % manager.ring, "all", "tile_records")]
        assert torch.equal(buffer[: len(active) * per].view(-1, per), records[active])
        assert torch.equal(buffer[E * per: E * per + len(active) * columns].view(-1, columns), cols[active])
    y, logits = streamed.forward_streaming(x, manager, 0)  # its own router
    assert (y.float() - resident(x, router_logits=logits)[0].float()).abs().max() <= 2e-2


def test_layers_with_output_scales_are_streamed_as_planes(lib):
    import trismoe_b200 as tm
    from trismoe_b200 import staging, synth

    shape = synth.LayerShape(256, 192, 8, 2, rank=96, group_size=32)
    layer = synth.synth_layer(shape, seed=6, keep_sparse_gmap=True)
    outs = []
    for scaled in (False, True):
        blk = tm.TrisSparseMoeBlock(256, 192, 8, 2, True)
        payloads = [dict(layer[n], compact3_use_block_gr=False) for n in ("gate", "up", "down")]
        if scaled:
            payloads[2].update(output_scale=torch.full((8, 256), 2.0, dtype=torch.float16), has_output_scale=True)
        blk.load_grouped_payloads(*payloads, layer["shared_gate"], layer["shared_up"], layer["shared_down"], layer["router_weight"], device="cuda")
        manager = staging.GroupedQGmapCPUStagingManager([blk])
        manager.initialize()
        assert ((0, "down") in manager._record_info) == (not scaled)
        x = synth.synth_activations(7, 256, seed=1).cuda().view(1, 7, 256)
        outs.append(blk.forward_streaming(x, manager, 0, router_logits=synth.synth_router_logits(7, 8, seed=2).cuda())[0].float())
    assert (outs[1] - 2 * outs[0]).abs().max() <= 2e-2 * outs[0].abs().max()


@pytest.mark.parametrize("rank,group", [(96, 32), (256, 128), (300, 64)])
def test_records_stay_inside_their_plan(lib, rank, group):
    """Built for one salient step and one row-scale slot fewer than the payload has: what is beyond that is left out, and nothing behind the
    buffers is written."""
    import trismoe_b200 as tm
    from trismoe_b200 import synth
    from trismoe_b200.qlinear_grouped import proj_view

    rng = np.random.default_rng(rank)
    raws = synth.raw_projection(rng, 3, 200, rank, group_size=group, p_salient=0.5)
    payload = tm.prepare_grouped_payload(synth.pack_projection(raws, "cpu", True, True), "cuda")
    view = tm._native.TrisProjView.from_buffer_copy(proj_view(payload))
    count, steps = int(lib.tris_tile_record_count(C.byref(view))), view.max_sal_words
    slots = min(4, -(-min(rank, 128) // group))
    assert steps >= 2
    for fewer_steps, fewer_slots in ((1, 0), (steps, 0), (0, min(1, slots - 1)), (steps, slots - 1)):
        n, size = steps - fewer_steps, proj_view(payload).max_record_bytes - 4 * (128 * fewer_steps + 256 * fewer_slots)
        columns = int(lib.tris_col_record_bytes(C.byref(view), n))
        records, cols = (torch.full((b + 8192,), 0xA5, dtype=torch.uint8, device="cuda") for b in (count * size, columns))
        view.max_record_bytes = size
        tm._native.check(lib.tris_tile_records_build(C.byref(view), payload["_tris_tile_desc"].data_ptr(), records.data_ptr(), cols.data_ptr(), n,
                                                     torch.cuda.current_stream().cuda_stream), "tile_records_build")
        assert bool((records[count * size:] == 0xA5).all()) and bool((cols[columns:] == 0xA5).all())
        # what does fit: the code words of every record are those of the whole plan
        if fewer_slots == 0:
            whole = payload["_tris_tile_records"][: count * (size + 512 * fewer_steps)].view(count, 4, -1)
            assert torch.equal(records[: count * size].view(count, 4, -1)[:, :, : size // 4 - 256 * slots], whole[:, :, : size // 4 - 256 * slots])


def test_paged_records_that_outgrow_their_plan_are_reported(lib):
    """Column maps edited in place after the buffers were laid out: more salient columns than the records have room for."""
    import trismoe_b200 as tm
    from trismoe_b200 import staging, synth

    shape = synth.LayerShape(256, 192, 8, 2, rank=96, group_size=32)
    layer = synth.synth_layer(shape, seed=6, keep_sparse_gmap=True)
    blk = tm.TrisSparseMoeBlock(256, 192, 8, 2, True)
    blk.load_grouped_payloads(*(dict(layer[n], compact3_use_block_gr=False) for n in ("gate", "up", "down")), layer["shared_gate"], layer["shared_up"],
                              layer["shared_down"], layer["router_weight"], device="cuda")
    manager = staging.GroupedQGmapCPUStagingManager([blk])
    manager.initialize()
    x = synth.synth_activations(7, 256, seed=1).cuda().view(1, 7, 256)
    blk.forward_streaming(x, manager, 0)
    assert blk.last_kernel_status() == 0
    blk._get_grouped_payload("down")["c_map"].fill_(-1)
    blk.forward_streaming(x, manager, 0)
    torch.cuda.synchronize()
    assert blk.last_kernel_status() == 4  # TRIS_ERR_CORRUPT


@pytest.mark.parametrize("name", ["output_scale", "bias"])
@pytest.mark.parametrize("mode,sparse", [("bitmap", True), ("payload", False)])
def test_a_scale_or_bias_given_after_initialisation_is_applied(lib, name, mode, sparse):
    """The same bits as a block that had it from the start, whose slots are read as planes, and those of before once it is taken away."""
    import trismoe_b200 as tm
    from trismoe_b200 import staging, synth
    from trismoe_b200.qlinear_grouped import proj_view

    layer = synth.synth_layer(synth.LayerShape(256, 192, 8, 2, rank=96, group_size=32), seed=6, keep_sparse_gmap=True)
    value = torch.linspace(0.5, 2.0, 8 * 256).view(8, 256).half()
    x, logits = synth.synth_activations(7, 256, seed=1).cuda().view(1, 7, 256), synth.synth_router_logits(7, 8, seed=2).cuda()

    def block(given):
        blk = tm.TrisSparseMoeBlock(256, 192, 8, 2, True)
        payloads = [{k: v.clone() if isinstance(v, torch.Tensor) else v for k, v in layer[n].items()} for n in ("gate", "up", "down")]
        for p in payloads:
            p["compact3_use_block_gr"] = not sparse
        if given:
            payloads[2].update({name: value.clone(), "has_" + name: True})
        blk.load_grouped_payloads(*payloads, layer["shared_gate"], layer["shared_up"], layer["shared_down"], layer["router_weight"], device="cuda")
        manager = staging.GroupedQGmapCPUStagingManager([blk], mode=mode)
        manager.initialize()
        return blk, manager, lambda: blk.forward_streaming(x, manager, 0, router_logits=logits)[0].clone()

    want = block(True)[2]()
    blk, manager, run = block(False)
    plain = run()
    dev_value = value.cuda()
    view = proj_view(blk._get_grouped_payload("down"))
    for _ in range(3):  # both ring places
        setattr(view, name, dev_value.data_ptr())
        assert torch.equal(run(), want)
    for _ in range(3):
        setattr(view, name, None)
        assert torch.equal(run(), plain)
    assert blk.last_kernel_status() == 0


@pytest.mark.parametrize("mode", ["bitmap", "payload"])
def test_layers_on_different_streams_share_a_manager(lib, mode):
    """Layers enqueued in turn on three streams with nothing but the manager's events between them: a place of the ring is written again
    while its last reader, on another stream, may still run.  The same bits as one after the other on one stream."""
    import trismoe_b200 as tm
    from trismoe_b200 import staging, synth

    H, I, E, k = 512, 384, 32, 4
    layer = synth.synth_layer(synth.LayerShape(H, I, E, k, rank=256, group_size=128), seed=9, keep_sparse_gmap=True)
    blk = tm.TrisSparseMoeBlock(H, I, E, k, True)
    payloads = [dict(layer[n], compact3_use_block_gr=mode == "payload") for n in ("gate", "up", "down")]
    blk.load_grouped_payloads(*payloads, layer["shared_gate"], layer["shared_up"], layer["shared_down"], layer["router_weight"], device="cuda")
    manager = staging.GroupedQGmapCPUStagingManager([blk], mode=mode)
    manager.collect_timings = False
    manager.initialize()
    xs = [synth.synth_activations(T, H, seed=i).cuda().view(1, T, H) for i, T in enumerate((40, 3, 64, 1, 24, 17))]
    logits = [synth.synth_router_logits(x.shape[1], E, seed=i).cuda() for i, x in enumerate(xs)]
    want = []
    for x, l in zip(xs, logits):
        want.append(blk.forward_streaming(x, manager, 0, router_logits=l)[0].clone())
        torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in range(3)], []
    for i in range(60):
        with torch.cuda.stream(streams[i % 3]):
            got.append(blk.forward_streaming(xs[i % 6], manager, 0, router_logits=logits[i % 6])[0])
    torch.cuda.synchronize()
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 6]), i
    assert blk.last_kernel_status() == 0
