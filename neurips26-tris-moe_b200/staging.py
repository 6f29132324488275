"""Streaming loader: expert payloads held in pinned host memory and paged to the GPU on a
side stream, overlapped with compute.

Role of ``GroupedQGmapCPUStagingManager`` (``grouped_payload_sidecar.py:764-1146`` in the
TriS-MoE tree), with two modes:

``mode="bitmap"``   what the reference streams: only the sparse grouping bitmap
                    ``q_gmap_sparse`` of every projection leaves the GPU (README:281-283), coded at
                    half its size; signs and scales stay resident.  Payloads must use the sparse bitmap
                    format (``compact3_use_block_gr = False``).
``mode="payload"``  every bulky per-expert tensor (sign planes, bitmap or block-GR stream and
                    its index, scale packs) lives in pinned host memory; only the small
                    tables (c_map, prefixes, offsets/meta, group table) stay resident.

Mechanism (differs from the reference on purpose).  The reference learns the active experts on
the host (a ``.cpu().tolist()`` of the route), then issues one ``copy_`` per expert range and
one kernel per chunk.  Here the copy is itself a kernel (``tris_page_experts``) that reads the
pinned buffers through their device mapping and is driven by the device-side route: it is
enqueued on a side stream right after the route kernel, copies exactly the active experts'
blocks into staging slot ``s`` = segment index, and writes the expert -> slot table the
grouped kernels index with.  Nothing is read back to the host.  Payloads without output scales
and biases are then built into tile records from the slots (``tris_moe_layer_forward_paged``: route,
pagers, builders and the rest of the layer in one native call), which the kernels of resident layers
read; the others are computed from the slots' planes.  Ordering is by events:
compute waits on "paged", the pager of the next use of a slot waits on "consumed".

Statistics: ``pipeline_stats`` counts calls and bytes as the reference's does (exact bytes
need the active expert count, which only the device knows, so ``bytes`` is an upper bound
from the slot count); :meth:`overlap_report` turns CUDA-event timings into the overlapped
fraction ``1 - stall / copy``.
"""
from __future__ import annotations

import contextlib
import ctypes as C
import threading
from typing import Optional

import torch

from . import _native
from ._native import TrisCodedPageJob, TrisPagedLayer, TrisPageJob, TrisPageLaunch, TrisProjView
from .qlinear_grouped import proj_view

BITMAP_KEYS = ("q_gmap_sparse",)
PAYLOAD_KEYS = ("qweight1", "qweight2_sparse", "q_gmap_sparse", "q_gmap_gr_words", "_tris_gr_index", "col_pack3", "row_pack3")
PROJECTIONS = ("gate", "up", "down")
MAX_PAGE_JOBS = 16  # TRIS_MAX_PAGE_JOBS of the C header
PAGE_BLOCK_BYTES = 1024  # TRIS_PAGE_BLOCK_BYTES


class _Entry:
    """One projection of one layer: pinned host tensors and their per-expert block sizes.  A sparse bitmap lies on the
    host in coded blocks (``tris_page_code_blocks``) where that makes it smaller."""

    def __init__(self, payload: dict, keys):
        self.payload = payload
        self.host = {}
        self.block_bytes = {}  # of an expert's block in a staging slot
        self.link_bytes = {}   # key -> of every expert's block on its way over the host link
        self.coded = {}        # key -> device offsets of the coded blocks
        self.rows = {}         # key -> second dimension of the tensor
        E = int(payload["qweight1"].shape[0])
        for key in keys:
            t = payload.get(key)
            if not isinstance(t, torch.Tensor) or t.numel() == 0:
                continue
            per = t.numel() // E * t.element_size()
            if per == 0:
                continue
            shape = list(t.shape)
            if per % 16:
                # only a 2-D stream (block-GR words) can be ragged: pad each expert's row with zeros
                if t.dim() != 2 or (16 % t.element_size()):
                    raise RuntimeError(f"trismoe_b200 staging: {key} has {per} bytes per expert, not a multiple of 16")
                step = 16 // t.element_size()
                shape[1] = (shape[1] + step - 1) // step * step
                per = shape[1] * t.element_size()
            self.block_bytes[key], self.link_bytes[key] = per, [per] * E
            if t.dim() > 1:
                self.rows[key] = int(shape[1])
            if key == "q_gmap_sparse" and t.is_cuda and self._code(key, t.contiguous(), E, per):
                continue
            host = torch.zeros(shape, dtype=t.dtype, pin_memory=True)
            host[tuple(slice(0, d) for d in t.shape)].copy_(t)
            self.host[key] = host

    def _code(self, key: str, t: torch.Tensor, experts: int, per: int) -> bool:
        """Codes a bitmap; False where the code would not be at least an eighth smaller."""
        if t.data_ptr() % 16 or experts * -(-per // PAGE_BLOCK_BYTES) * 64 > 0x7FFFFFFF:
            return False
        lib, blocks = _native.load(), -(-per // PAGE_BLOCK_BYTES)
        offsets = torch.zeros((experts * blocks + 1,), dtype=torch.int32, device=t.device)
        with torch.cuda.device(t.device):
            stream = torch.cuda.current_stream(t.device).cuda_stream
            units = torch.empty((experts * blocks,), dtype=torch.int32, device=t.device)
            _native.check(lib.tris_page_code_blocks(t.data_ptr(), per, experts, units.data_ptr(), None, None, stream), "page_code_blocks")
            torch.cumsum(units, 0, dtype=torch.int32, out=offsets[1:])
            ends = offsets[::blocks].tolist()  # waits
            if ends[-1] * 16 * 8 > experts * per * 7:
                return False
            # straight into pinned memory: streaming is for GPUs that have no room for another copy
            host = torch.empty((max(1, ends[-1]) * 16,), dtype=torch.uint8, pin_memory=True)
            _native.check(lib.tris_page_code_blocks(t.data_ptr(), per, experts, None, offsets.data_ptr(), host.data_ptr(), stream), "page_code_blocks")
            torch.cuda.current_stream(t.device).synchronize()
        self.host[key], self.coded[key] = host, offsets
        self.link_bytes[key] = [16 * (hi - lo) for lo, hi in zip(ends, ends[1:])]
        return True


def staging_requested() -> bool:
    """True when the host asks for the streaming mode through ``TRIS_GROUPED_QGMAP_CPU_STAGING`` (or
    the reference's per-family names; ``_grouped_qgmap_cpu_staging_enabled``,
    grouped_payload_sidecar.py:147-152)."""
    from . import envflags

    return envflags.grouped_qgmap_cpu_staging_enabled()


class GroupedQGmapCPUStagingManager:
    """Pages expert payloads of the registered MoE blocks from pinned host memory."""

    def __init__(self, moe_blocks, mode: str = "bitmap", max_active_experts: Optional[int] = None, slots: int = 2):
        if mode not in ("bitmap", "payload"):
            raise ValueError("mode must be 'bitmap' or 'payload'")
        self.blocks = list(moe_blocks)
        self.mode = mode
        self.ring = int(slots)
        self.max_active = max_active_experts
        self.device = None
        self.entries = {}          # (block index, projection) -> _Entry
        self.buffers = {}          # (ring slot, projection, key) -> device staging tensor
        self.slot_tables = []      # per ring slot: {"gate" (shared with up), "down"}: int32 [E] expert -> staging
                                   # slot; down has its own because each pager call resets its table and down is
                                   # paged while the gate/up kernel is still reading the table of gate and up
        self._paged = []           # per ring slot: event "pager done" (all three projections)
        self._paged_gu = []        # per ring slot: event "gate and up paged" (down may still be in flight)
        self._plans = {}           # (layer, ring slot) -> pager jobs and staged views: host and slot addresses are fixed
        self._consumed = []        # per ring slot: event "compute done with this slot"
        self._used = []
        self._copy_stream = None
        self._next = 0
        self._lock = threading.RLock()
        self._initialized = False
        # bytes: at most, as if every slot of a launch were used and by the largest expert
        self.pipeline_stats = {"calls": 0, "chunks": 0, "bytes": 0, "slot_reuses": 0}
        self._timings = []         # (copy_start, copy_end, wait_start, wait_end) events
        self.collect_timings = True  # set False while capturing the forward into a CUDA graph
        # A stream that is being captured may not wait for an event recorded outside the
        # capture.  Slot uses are therefore stamped with an epoch that changes whenever a
        # capture starts or ends; a pager only waits for "consumed" events of its own epoch
        # (work of an earlier epoch is ordered before it by the stream itself: the caller
        # captures, and replays, on the stream the earlier work ran on or has synchronised).
        self._epoch = 0
        self._capturing = False
        self._consumed_epoch = []
        self._route_done = None
        self._record_info = {}     # (block index, projection) -> sizes of the tile records of its paged experts
        self._record_keys = {}     # block index -> what they were planned for
        self._record_bytes = 0     # of an expert, at most
        self._slot_ids = None
        self._layers = {}          # (layer, ring slot) -> what the native layer call takes: TrisPagedLayer and what it points at

    @property
    def buffer_nbytes(self) -> int:
        return sum(t.numel() * t.element_size() for t in self.buffers.values())

    def initialize(self) -> bool:
        with self._lock:  # of several threads' first calls one lays the buffers out
            return self._initialized or self._initialize()

    def _initialize(self) -> bool:
        if not self.blocks:
            return False
        keys = BITMAP_KEYS if self.mode == "bitmap" else PAYLOAD_KEYS
        first = self.blocks[0]._get_grouped_payload("gate")
        self.device = first["qweight1"].device
        if self.device.type != "cuda":
            raise RuntimeError("trismoe_b200 staging: payloads must be on a CUDA device before staging starts")
        E = int(first["qweight1"].shape[0])
        cap = E if self.max_active is None else max(1, min(E, int(self.max_active)))
        sizes = {}
        for bi, blk in enumerate(self.blocks):
            for proj in PROJECTIONS:
                payload = blk._get_grouped_payload(proj)
                if payload["qweight1"].device != self.device:
                    raise RuntimeError("trismoe_b200 staging: all layers must live on one CUDA device")
                if self.mode == "bitmap" and bool(payload.get("compact3_use_block_gr", False)):
                    raise RuntimeError("trismoe_b200 staging: bitmap streaming needs the sparse bitmap format "
                                       "(block-GR payloads stay resident, as in the reference)")
                entry = _Entry(payload, keys)
                self.entries[(bi, proj)] = entry
                for key, per in entry.block_bytes.items():
                    sizes[(proj, key)] = max(sizes.get((proj, key), 0), per)
        for ring in range(self.ring):
            for (proj, key), per in sizes.items():
                # a few bytes of slack: the GR span copy may round its end up to 16 bytes
                self.buffers[(ring, proj, key)] = torch.zeros((cap * per + 64,), dtype=torch.uint8, device=self.device)
            self.slot_tables.append({proj: torch.full((E,), -1, dtype=torch.int32, device=self.device) for proj in ("gate", "down")})
            self._paged.append(torch.cuda.Event())
            self._paged_gu.append(torch.cuda.Event())
            self._consumed.append(torch.cuda.Event())
            self._used.append(False)
            self._consumed_epoch.append(-1)
        self._copy_stream = torch.cuda.Stream(device=self.device)
        self.capacity = cap
        self._route_done = torch.cuda.Event()
        for event in (*self._paged, *self._paged_gu, *self._consumed, self._route_done):
            event.record(self._copy_stream)  # an event has its handle from then on
        self._plan_records(E, cap)
        # drop the device copies: from here on the tensors exist only in pinned host memory
        for entry in self.entries.values():
            for key in entry.host:
                entry.payload[key] = torch.empty((0,), dtype=entry.payload[key].dtype, device=self.device)
            if self.mode == "payload":
                # the resident tile-major copy of the same planes would defeat the point of paging them
                for key in ("_tris_tile_records", "_tris_tile_desc", "_tris_col_records", "_tris_tile_meta"):
                    entry.payload.pop(key, None)
                view = proj_view(entry.payload)
                view.tile_records = view.tile_desc = view.col_records = None
            entry.payload["_qgmap_staging"] = (self, entry)
        self._initialized = True
        return True

    @staticmethod
    def _record_key(views):
        """What the sizes of a layer's records, and whether it may have any, follow from."""
        return tuple((v.num_experts, v.out_features, v.rank, v.num_groups, v.use_block_gr, v.gr_substreams, v.c_map, v.packed_row_group, v.output_scale,
                      v.bias) for v in views)

    def _plan_block(self, block_index: int) -> int:
        """Sizes of the tile records of one expert of a layer; returns the bytes of them, gate and up or down.  0: none, the layer is
        computed from the planes.  Waits for the GPU."""
        lib = _native.load()
        views = [proj_view(self.entries[(block_index, proj)].payload) for proj in PROJECTIONS]
        self._record_keys[block_index] = self._record_key(views)
        for proj in PROJECTIONS:
            self._record_info.pop((block_index, proj), None)
        # a record's place is that of its segment, which output scales and biases are not indexed by
        if any(v.output_scale or v.bias or (v.use_block_gr and v.gr_substreams != 32) for v in views):
            return 0
        with torch.cuda.device(self.device):
            stream = torch.cuda.current_stream(self.device).cuda_stream
            info = torch.zeros((3, 4), dtype=torch.int64, device=self.device)
            for i, v in enumerate(views):
                _native.check(lib.tris_paged_records_plan(C.byref(v), info[i].data_ptr(), stream), "paged_records_plan")
            for proj, v, (per, size, steps, _) in zip(PROJECTIONS, views, info.tolist()):
                one = TrisProjView()
                C.pointer(one)[0] = v
                one.num_experts = 1
                columns = int(lib.tris_col_record_bytes(C.byref(one), steps))
                self._record_info[(block_index, proj)] = (per, size, steps, columns)
        gate, up, down = (sum(self._record_info[(block_index, proj)][i] for i in (0, 3)) for proj in PROJECTIONS)
        return max(gate + up, down)

    def _plan_records(self, experts: int, cap: int) -> None:
        """Buffers for the tile records of the experts of one layer, gate and up or down, per ring slot: the grouped kernels for records
        are about twice as fast as those that read the planes, and building records from paged planes takes a fraction of that."""
        self._record_bytes = max(self._plan_block(bi) for bi in range(len(self.blocks)))
        if self._record_bytes:
            for ring in range(self.ring):
                self.buffers[(ring, "all", "tile_records")] = torch.empty((cap * self._record_bytes,), dtype=torch.uint8, device=self.device)
            ids = torch.arange(max(experts, cap), dtype=torch.int32, device=self.device)
            self._slot_ids = torch.where(ids < cap, ids, torch.full_like(ids, -1))

    def _has_records(self, block_index: int) -> bool:
        """Whether a layer's experts become tile records: not with output scales or biases, which a view may have been given after the
        buffers were laid out, and not where the records of the view's present tables would not fit the buffers."""
        views = [proj_view(self.entries[(block_index, proj)].payload) for proj in PROJECTIONS]
        if self._record_keys.get(block_index) != self._record_key(views):
            if torch.cuda.is_current_stream_capturing():
                return False  # planning waits for the GPU
            if self._plan_block(block_index) > self._record_bytes:
                for proj in PROJECTIONS:
                    del self._record_info[(block_index, proj)]
        return (block_index, "gate") in self._record_info

    # -- one layer ---------------------------------------------------------------------------
    @contextlib.contextmanager
    def native_layer(self, block_index: int, rows: int, experts: int):
        """The argument of ``tris_moe_layer_forward_paged`` for a layer that routes ``rows`` rows, for the length of that call: takes a
        ring slot as :meth:`page_layer` does, which is in use afterwards until its "consumed" event, recorded by the call.  Other
        threads wait meanwhile: the argument, the events and the order of the copy stream are the manager's."""
        with self._lock:
            self.initialize()
            ring = self._take_slot()
            launches, views = self._plan(block_index, ring)
            layer = self._layers.get((block_index, ring))
            if layer is None or layer[0] is not launches:
                layer = self._layers[(block_index, ring)] = (launches, *self._paged_layer(block_index, ring, launches, views))
            arg = layer[1]
            arg.wait_consumed = int(self._used[ring] and self._consumed_epoch[ring] == self._epoch)
            self.pipeline_stats["slot_reuses"] += arg.wait_consumed
            nseg_bound = min(experts, rows, self.capacity)
            self.pipeline_stats["bytes"] += nseg_bound * sum(launch[3] for launch in launches)
            self.pipeline_stats["chunks"] += len(launches)
            self.pipeline_stats["calls"] += 1
            if self.collect_timings:
                compute = torch.cuda.current_stream(self.device)
                events = [torch.cuda.Event(enable_timing=True) for _ in range(6)]
                for event in events:
                    event.record(compute)  # an event has its handle from then on; recorded again by the call
                arg.timing[:] = [event.cuda_event for event in events]
                begin, end, w0, w1, w2, w3 = events
                self._timings += [(begin, end, w0, w1), (w2, w2, w2, w3)]
            else:
                arg.timing[:] = [None] * 6
            yield arg
            self._used[ring] = True
            self._consumed_epoch[ring] = self._epoch

    def _paged_layer(self, block_index: int, ring: int, launches, views):
        arg, keep = TrisPagedLayer(), []
        groups, group = ([], []), 0
        for coded, jobs, count, _, last_of_gate_up, table in launches:
            groups[group].append(TrisPageLaunch(C.addressof(jobs), table, count, int(coded)))
            group += int(last_of_gate_up)
        for g, group in enumerate(groups):
            pages = (TrisPageLaunch * max(1, len(group)))(*group)
            keep.append(pages)
            arg.pages[g], arg.num_pages[g] = C.addressof(pages), len(group)
        records = self.buffers.get((ring, "all", "tile_records")) if self._has_records(block_index) else None
        at = 0
        for i, proj in enumerate(PROJECTIONS):
            arg.staged[i] = views[proj]
            if records is None:
                continue
            arg.records[i] = proj_view(self.entries[(block_index, proj)].payload)
            per, size, steps, columns = self._record_info[(block_index, proj)]
            rec, at = arg.records[i], at if proj != "down" else 0  # down's take the place of gate's and up's, which are done with
            rec.num_experts, rec.use_block_gr, rec.gmap_slot, rec.expert_slot = self.capacity, 1, None, None
            rec.max_record_bytes, rec.max_sal_words = size, steps
            rec.col_record_bytes = columns // max(1, per // (size * -(-rec.out_features // 128)))
            rec.tile_records, rec.col_records = records.data_ptr() + at, records.data_ptr() + at + self.capacity * per
            at += self.capacity * (per + columns)
        arg.slot_ids, arg.capacity = None if self._slot_ids is None else self._slot_ids.data_ptr(), self.capacity
        arg.copy_stream, arg.event_route = self._copy_stream.cuda_stream, self._route_done.cuda_event
        arg.event_paged[:] = [self._paged_gu[ring].cuda_event, self._paged[ring].cuda_event]
        arg.event_consumed = self._consumed[ring].cuda_event
        return arg, keep

    def _take_slot(self) -> int:
        with self._lock:
            ring = self._next
            self._next = (self._next + 1) % self.ring
            capturing = bool(torch.cuda.is_current_stream_capturing())
            if capturing != self._capturing:
                self._capturing = capturing
                self._epoch += 1
            return ring

    def page_layer(self, block_index: int, route: dict):
        """Enqueues, on the side stream, the paging of gate/up/down of one layer for the
        experts of ``route`` (device arrays from ``tris_build_grouped_route``), and returns a
        handle whose views the grouped kernels of this layer must use."""
        self.initialize()
        lib = _native.load()
        compute = torch.cuda.current_stream(self.device)
        copy = self._copy_stream
        copy.wait_stream(compute)  # the route must be final before the pager reads it
        ring = self._take_slot()
        if self._used[ring] and self._consumed_epoch[ring] == self._epoch:
            copy.wait_event(self._consumed[ring])
            self.pipeline_stats["slot_reuses"] += 1
        nseg_bound = min(int(route["experts"]), int(route["rows"]), self.capacity)
        timed = self.collect_timings
        start = end = None
        if timed:
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        launches, views = self._plan(block_index, ring)
        ids, counts, experts = route["expert_ids"], route["counts"], int(route["experts"])
        ids, counts = (v if isinstance(v, int) else v.data_ptr() for v in (ids, counts))  # tensors or device addresses
        with torch.cuda.stream(copy):
            if timed:
                start.record(copy)
            # gate and up go in one launch (they are needed together and share a slot table), down in a second one
            # that runs while the gate/up kernel computes
            for coded, jobs, count, per_segment, last_of_gate_up, table in launches:
                self.pipeline_stats["bytes"] += nseg_bound * per_segment
                page = lib.tris_page_coded_experts if coded else lib.tris_page_experts
                _native.check(page(jobs, count, ids, counts, nseg_bound, experts, table, copy.cuda_stream), "page_experts")
                self.pipeline_stats["chunks"] += 1
                if last_of_gate_up:  # the gate/up kernel may start while down is still paged
                    self._paged_gu[ring].record(copy)
            if timed:
                end.record(copy)
            self._paged[ring].record(copy)
        self.pipeline_stats["calls"] += 1
        self._used[ring] = True
        return _PagedLayer(self, ring, views, start, end)

    def _plan(self, block_index: int, ring: int):
        """Pager launches ``(coded, jobs, count, most bytes per segment, ends gate/up, slot table)`` and staged views of a
        layer in a ring slot, laid out on first use and again when a projection's own view has other contents
        (an object's identity would miss a view edited in place, and one built at a freed view's address)."""
        bases = tuple(bytes(proj_view(self.entries[(block_index, proj)].payload)) for proj in PROJECTIONS)
        plan = self._plans.get((block_index, ring))
        if plan is not None and plan[0] == bases:
            return plan[1], plan[2]
        launches, views = [], {}
        for group in (("gate", "up"), ("down",)):
            table, parts = self.slot_tables[ring][group[0]], []
            pages = [(proj, key, self.entries[(block_index, proj)]) for proj in group for key in self.entries[(block_index, proj)].host]
            for coded in (False, True):
                these = [page for page in pages if (page[1] in page[2].coded) == coded]
                parts += [(coded, these[lo: lo + MAX_PAGE_JOBS]) for lo in range(0, len(these), MAX_PAGE_JOBS)]
            for i, (coded, part) in enumerate(parts):
                jobs = ((TrisCodedPageJob if coded else TrisPageJob) * len(part))()
                for job, (proj, key, entry) in zip(jobs, part):
                    job.host_src = entry.host[key].data_ptr()
                    job.dst = self.buffers[(ring, proj, key)].data_ptr()
                    job.bytes_per_expert = entry.block_bytes[key]
                    if coded:
                        job.block_offsets = entry.coded[key].data_ptr()
                per_segment = sum(max(entry.link_bytes[key]) for _, key, entry in part)
                launches.append((coded, jobs, len(part), per_segment, group[0] == "gate" and i + 1 == len(parts), table.data_ptr()))
            for proj in group:
                views[proj] = self._staged_view(self.entries[(block_index, proj)], ring, proj, table)
        self._plans[(block_index, ring)] = (bases, launches, views)
        return launches, views

    def _staged_view(self, entry: _Entry, ring: int, proj: str, table: torch.Tensor):
        """Copy of the projection's ctypes view whose paged tensors point at the staging slots."""
        base = proj_view(entry.payload)
        view = type(base)()
        C.pointer(view)[0] = base
        field = {"qweight1": "qweight1", "qweight2_sparse": "qweight2_sparse", "q_gmap_sparse": "q_gmap_sparse",
                 "q_gmap_gr_words": "q_gmap_gr_words", "_tris_gr_index": "gr_index", "col_pack3": "col_pack3",
                 "row_pack3": "row_pack3"}
        for key in entry.host:
            setattr(view, field[key], self.buffers[(ring, proj, key)].data_ptr())
        if self.mode == "bitmap":
            view.gmap_slot = table.data_ptr()
            view.gmap_sparse_rows = entry.rows["q_gmap_sparse"]
        else:
            view.expert_slot = table.data_ptr()
            if "q_gmap_sparse" in entry.host:
                view.gmap_sparse_rows = entry.rows["q_gmap_sparse"]
            if "q_gmap_gr_words" in entry.host:
                view.gr_max_words = entry.rows["q_gmap_gr_words"]
        return view

    # -- reporting -----------------------------------------------------------------------------
    def overlap_report(self) -> dict:
        """Overlapped fraction of the transfer time: 1 - (time compute stalled on a pager) /
        (pager time), from CUDA events; call after a synchronize."""
        copy_ms = stall_ms = 0.0
        n = 0
        for c0, c1, w0, w1 in self._timings:
            if c0 is not c1:  # a layer's second wait carries no copy interval of its own
                copy_ms += c0.elapsed_time(c1)
                n += 1
            stall_ms += w0.elapsed_time(w1)
        self._timings = []
        frac = 1.0 - stall_ms / copy_ms if copy_ms > 0 else None
        return {"layers": n, "copy_ms": copy_ms, "stall_ms": stall_ms, "overlapped_fraction": frac}

    def finalize_forward(self) -> None:
        """Kept for interface parity (grouped_payload_sidecar.py:1143): nothing to unbind."""


class _PagedLayer:
    def __init__(self, manager: GroupedQGmapCPUStagingManager, ring: int, views: dict, start, end):
        self.manager, self.ring, self.views = manager, ring, views
        self._copy_start, self._copy_end = start, end
        self._waited = False
        self._waited_gu = False

    def wait(self, which: str = "all") -> None:
        """Makes the current (compute) stream wait for this layer's pager, timing the stall.
        ``which="gate_up"`` waits only until gate and up are in (the pager goes on with down, which
        then pages under the gate/up kernel and the down backbone); ``"all"`` waits for everything."""
        if self._waited or (which == "gate_up" and self._waited_gu):
            return
        compute = torch.cuda.current_stream(self.manager.device)
        event = self.manager._paged_gu[self.ring] if which == "gate_up" else self.manager._paged[self.ring]
        if self._copy_start is None:
            compute.wait_event(event)
        else:
            w0, w1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            w0.record(compute)
            compute.wait_event(event)
            w1.record(compute)
            # the copy interval is counted once (with the first wait), every wait adds its stall
            zero = (w0, w0) if (self._waited_gu and which != "gate_up") else (self._copy_start, self._copy_end)
            self.manager._timings.append((zero[0], zero[1], w0, w1))
        if which == "gate_up":
            self._waited_gu = True
        else:
            self._waited = True

    def release(self) -> None:
        """Marks the staging slots free once the kernels enqueued so far have consumed them."""
        self.manager._consumed[self.ring].record(torch.cuda.current_stream(self.manager.device))
        self.manager._consumed_epoch[self.ring] = self.manager._epoch


def maybe_create_grouped_qgmap_cpu_staging_manager(moe_blocks, mode: str = "bitmap", **kw):
    """``maybe_create_grouped_qgmap_cpu_staging_manager`` (grouped_payload_sidecar.py:1149-1153)."""
    manager = GroupedQGmapCPUStagingManager(moe_blocks, mode=mode, **kw)
    return manager if manager.initialize() else None
