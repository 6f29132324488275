"""CPU tests of the pager plan of a layer: what it launches, and that a cached one follows the projections' own views."""
import contextlib
import ctypes as C
import threading
import types

import pytest
import torch


def _manager(tm, staging, coded=()):
    man = staging.GroupedQGmapCPUStagingManager([], mode="bitmap")
    man.slot_tables = [{p: torch.zeros((4,), dtype=torch.int32) for p in ("gate", "down")}]
    for proj in staging.PROJECTIONS:
        host, key = torch.zeros((4, 2, 8), dtype=torch.int32), "q_gmap_sparse"
        view = tm._native.TrisProjView()
        view.out_features, view.output_scale = 8, 4096
        # all that an entry has but pinned memory, which needs a GPU
        man.entries[(0, proj)] = types.SimpleNamespace(payload={"_tris_prepared": True, "_tris_view": view}, host={key: host}, block_bytes={key: 64},
                                                       link_bytes={key: [16, 32, 0, 16] if proj in coded else [64] * 4}, rows={key: 2},
                                                       coded={key: torch.zeros((5,), dtype=torch.int32)} if proj in coded else {})
        man.buffers[(0, proj, "q_gmap_sparse")] = torch.zeros((64,), dtype=torch.uint8)
    return man


@pytest.mark.parametrize("proj", ["gate", "up", "down"])
def test_plan_follows_a_view_that_is_rebuilt_or_edited(proj):
    import trismoe_b200 as tm
    from trismoe_b200 import staging

    man = _manager(tm, staging)
    launches, views = man._plan(0, 0)
    again = man._plan(0, 0)
    assert again[0] is launches and again[1] is views and views[proj].output_scale == 4096
    payload = man.entries[(0, proj)].payload
    payload["_tris_view"].output_scale = 8192  # in place
    assert man._plan(0, 0)[1][proj].output_scale == 8192
    # rebuilt until an address comes back that an earlier, freed view had
    seen = {id(payload["_tris_view"])}
    for i in range(1, 2000):
        payload["_tris_view"] = None
        view = tm._native.TrisProjView()
        view.out_features, view.output_scale = 8, 4096 * (2 + i)
        payload["_tris_view"] = view
        assert man._plan(0, 0)[1][proj].output_scale == 4096 * (2 + i)
        if id(view) in seen:
            break
        seen.add(id(view))
    else:
        pytest.skip("no address was used twice")


@pytest.mark.parametrize("coded", [(), ("gate",), ("up",), ("gate", "up"), ("down",), ("gate", "up", "down")])
def test_raw_and_coded_tensors_go_in_launches_of_their_own(coded):
    """One launch per kind and group, raw before coded; the last one of gate and up ends the group, none of down does."""
    import trismoe_b200 as tm
    from trismoe_b200 import staging

    man = _manager(tm, staging, coded)
    launches, views = man._plan(0, 0)
    want = [(kind, procs) for group in (("gate", "up"), ("down",)) for kind in (False, True)
            for procs in [[p for p in group if (p in coded) == kind]] if procs]
    assert [(kind, count) for kind, _, count, _, _, _ in launches] == [(kind, len(procs)) for kind, procs in want]
    last_gate_up = max(i for i, (_, procs) in enumerate(want) if "down" not in procs)
    for i, ((kind, jobs, count, most, ends, table), (_, procs)) in enumerate(zip(launches, want)):
        assert isinstance(jobs, C.Array) and isinstance(jobs[0], tm._native.TrisCodedPageJob if kind else tm._native.TrisPageJob)
        assert most == (32 if kind else 64) * count and ends == (i == last_gate_up)
        assert table == man.slot_tables[0][procs[0] if procs[0] == "down" else "gate"].data_ptr()
        for job, proj in zip(jobs, procs):
            entry = man.entries[(0, proj)]
            assert job.host_src == entry.host["q_gmap_sparse"].data_ptr() and job.bytes_per_expert == 64
            assert job.dst == man.buffers[(0, proj, "q_gmap_sparse")].data_ptr()
            assert not kind or job.block_offsets == entry.coded["q_gmap_sparse"].data_ptr()
    for proj in staging.PROJECTIONS:
        assert views[proj].q_gmap_sparse == man.buffers[(0, proj, "q_gmap_sparse")].data_ptr() and views[proj].gmap_sparse_rows == 2


def test_threads_that_stream_at_once_take_places_of_their_own(monkeypatch):
    """The native call gives up the interpreter lock: a layer of another thread that comes in meanwhile changes nothing of the argument, and
    each marks its own place of the ring as used."""
    import trismoe_b200 as tm
    from trismoe_b200 import staging

    man = _manager(tm, staging)
    man._initialized, man.device, man.capacity, man.ring, man.collect_timings = True, torch.device("cpu"), 4, 2, False
    man.slot_tables = man.slot_tables * 2
    man.buffers.update({(1, proj, key): t for (_, proj, key), t in list(man.buffers.items())})
    man._used, man._consumed_epoch = [False, False], [-1, -1]
    man._paged_layer = lambda bi, ring, launches, views: (types.SimpleNamespace(ring=ring, wait_consumed=0, timing=[None] * 6), [])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(tm._native, "on_device", lambda dev: contextlib.nullcontext())
    monkeypatch.setattr(tm._native, "stream_of", lambda dev: 0)
    monkeypatch.setattr(C, "byref", lambda v: v)
    calls, others, inside = [], [], threading.Event()

    def forward_paged(view, paged, *rest):
        seen = (paged.ring, paged.wait_consumed)
        if not others:  # the first call: another thread's layer comes in before this one returns
            others.append(threading.Thread(target=forward))
            others[0].start()
            inside.wait(0.5)  # runs out where the other one has to wait
        else:
            inside.set()
        calls.append((seen, (paged.ring, paged.wait_consumed)))
        return 0

    lib = types.SimpleNamespace(tris_moe_layer_workspace_bytes=lambda view, tokens: 64, tris_moe_layer_forward_paged=forward_paged)
    status = torch.zeros((1,), dtype=torch.int32)
    blk = types.SimpleNamespace(num_experts=4, top_k=2, layer_view=lambda: None, _status_of=lambda dev: status)
    x = torch.zeros((3, 8), dtype=torch.float16)
    forward = lambda: tm.TrisSparseMoeBlock._forward_streaming_native(blk, lib, x, x.clone(), man, 0, torch.zeros((3, 4)))
    forward()
    others[0].join()
    assert all(before == after for before, after in calls) and sorted(ring for (ring, _), _ in calls) == [0, 1]
    assert man._used == [True, True] and man._consumed_epoch == [man._epoch] * 2
    forward()
    assert calls[-1][0] == (0, 1)  # waits for the last use of its place
