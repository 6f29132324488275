"""MoE block on the trismoe_b200 runtime, mirroring ``OlmoeSparseMoeBlock``
(``auto_gptq/modeling_tris_moe/modeling_olmoe.py:621-1105`` in the TriS-MoE tree; the
Mixtral and Qwen2-MoE blocks call the same operators with other shapes).

``forward`` runs the whole block through one C-ABI call (``tris_moe_layer_forward``):
router, route, both input-side backbones, grouped gate/up with SiLU*mul, down backbone,
grouped down and the weighted combine, stream-ordered with no host synchronisation.
``forward_grouped_ops`` composes the same result from the individual reference-named
operators, the way ``_forward_grouped`` (modeling_olmoe.py:916-1044) does.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch
from torch import nn

from . import _native, envflags
from ._native import TrisMoeLayerExtras, TrisMoeLayerView, TrisSharedExpert
from .ns_compensation import Packed4Linear
from .qlinear_grouped import (
    build_grouped_route,
    compute_shared_hidden,
    dequantize_packed_4bit,
    prepare_grouped_payload,
    proj_view,
    run_grouped_structured_expert_forward,
    run_grouped_structured_expert_pair_forward,
)


class TrisSparseMoeBlock(nn.Module):
    """Quantized grouped-expert MoE layer.

    Args mirror the HF config fields the reference block reads: ``hidden_size``,
    ``intermediate_size``, ``num_experts``, ``num_experts_per_tok``, ``norm_topk_prob``.
    Weights are attached with :meth:`load_grouped_payloads`.
    """

    def __init__(self, hidden_size: int, intermediate_size: int, num_experts: int, num_experts_per_tok: int,
                 norm_topk_prob: bool = False):
        super().__init__()
        self.hidden_size = int(hidden_size)
        self.intermediate_size = int(intermediate_size)
        self.num_experts = int(num_experts)
        self.top_k = int(num_experts_per_tok)
        self.norm_topk_prob = bool(norm_topk_prob)
        self.gate = nn.Linear(self.hidden_size, self.num_experts, bias=False, dtype=torch.float16)
        self.register_buffer("shared_gate", torch.zeros((0, 0), dtype=torch.float16))
        self.register_buffer("shared_up", torch.zeros((0, 0), dtype=torch.float16))
        self.register_buffer("shared_down", torch.zeros((0, 0), dtype=torch.float16))
        self.packed_backbones: dict = {}  # name -> Packed4Linear: backbones kept in their 4-bit nibbles
        self.input_scales: dict = {}      # name -> fp16 [in]: vector null-space input scale (ns_mode == 1)
        self.ns_payloads: dict = {}       # name -> grouped null-space compensation payload (ns_mode == 2)
        self._grouped_payload_cache: dict = {}
        self._layer_view: Optional[TrisMoeLayerView] = None
        self._expanded_view: Optional[dict] = None  # expanded backbone names -> layer view
        self._workspace: Optional[torch.Tensor] = None
        self._workspace_for = None
        self._status_word: Optional[torch.Tensor] = None  # see _status_of

    # -- loading ---------------------------------------------------------------------------
    # Activation rows above which a 4-bit backbone is expanded to fp16 scratch and run on the dense GEMM.  One matrix on
    # B200, 4-bit GEMM against expansion and GEMM in us: 256 x 2048 6.8 / 7.0 at 1 row, 8.1 / 9.3 at 32, 11.2 / 9.9 at
    # 64, 13.2 / 12.4 at 1024; 256 x 1024 4.7 / 6.4 at 16, 7.5 / 9.0 at 128, 8.8 / 11.0 at 1024; 256 x 4096 13.3 / 9.9 at
    # 16; 256 x 14336 38 / 18 at 1.  So 64 rows is right for 2048 columns; fewer columns would rather stay packed up to
    # some 1000 rows (by 1.5 us), more columns rather be expanded from the first row on.
    PACKED_BACKBONE_MAX_ROWS = 64
    _expand_scratch: dict = {}  # (device, name, shape) -> fp16 scratch shared by every block of a model

    def load_grouped_payloads(self, gate: dict, up: dict, down: dict, shared_gate, shared_up, shared_down,
                              router_weight: Optional[torch.Tensor] = None, device=None,
                              packed_backbone: Optional[str] = None, input_scales: Optional[dict] = None) -> "TrisSparseMoeBlock":
        """Attaches the E-stacked payloads (``enable_grouped_deployment_only``,
        modeling_olmoe.py:732-804) and the three backbones, moving everything to ``device`` and
        deriving the decode index once.  A backbone is an fp16 matrix ``[r, in]`` or, as real
        checkpoints store it, a 4-bit packed payload dict (``shared_sv_quant``: ``qweight``, ``qzeros``,
        ``scales``, ``g_idx``, ``rows``, ``cols``).  ``packed_backbone`` (default: the environment
        variable ``TRIS_PACKED4_BACKBONE``, else ``"nibbles"``) says how packed backbones are kept:
        ``"nibbles"`` - in place, read by the 4-bit GEMM (a quarter of the bytes; gate and up switch
        together, matrices with non-uniform groups are expanded), ``"fp16"`` - expanded once at load.
        ``input_scales`` (``{"gate" | "up" | "down": fp16 [in]}``): the vector null-space input scale of
        ``ns_mode == 1`` checkpoints (``expert_input_scale`` of expert 0, qlinear_cuda.py:3918-3923): the
        backbone of that projection sees ``x * scale`` rounded to fp16 (qlinear_cuda.py:4477-4480); the
        matching output scale travels in the payload (``output_scale``).  A scaled projection's
        backbone is a launch of its own (gate and up no longer share their input rows)."""
        import os

        dev = torch.device(device) if device is not None else gate["qweight1"].device
        self._grouped_payload_cache = {
            "gate": prepare_grouped_payload(gate, dev),
            "up": prepare_grouped_payload(up, dev),
            "down": prepare_grouped_payload(down, dev),
        }
        mode = (packed_backbone or os.environ.get("TRIS_PACKED4_BACKBONE", "nibbles")).lower()
        if mode not in ("nibbles", "fp16"):
            raise ValueError("packed_backbone must be 'nibbles' or 'fp16'")
        given = {"gate": shared_gate, "up": shared_up, "down": shared_down}
        is_packed = {n: isinstance(m, dict) and "qweight" in m for n, m in given.items()}
        keep = {n: mode == "nibbles" and is_packed[n] and Packed4Linear.supports(m) for n, m in given.items()}
        keep["gate"] = keep["up"] = keep["gate"] and keep["up"]
        self.packed_backbones = {}
        for name, m in given.items():
            if keep[name]:
                self.packed_backbones[name] = Packed4Linear(m, dev)
                dense = torch.zeros((0, 0), dtype=torch.float16, device=dev)
            elif is_packed[name]:
                dense = dequantize_packed_4bit(m, dev)
            else:
                dense = m.to(dev, torch.float16).contiguous()
            setattr(self, "shared_" + name, dense)
        if router_weight is not None:
            self.gate.weight = nn.Parameter(router_weight.to(dev, torch.float16).contiguous(), requires_grad=False)
        else:
            self.gate.to(dev)
        self.input_scales = {n: v.reshape(-1).to(dev, torch.float16).contiguous() for n, v in (input_scales or {}).items()}
        if set(self.input_scales) - set(given):
            raise ValueError("input_scales keys must be among 'gate', 'up', 'down'")
        if self.input_scales:
            self._status_of(dev)  # made here and not by the first of several threads
        self._layer_view = self._expanded_view = None
        return self

    def load_ns_compensation_payloads(self, gate_ns: Optional[dict] = None, up_ns: Optional[dict] = None,
                                      down_ns: Optional[dict] = None) -> "TrisSparseMoeBlock":
        """Attaches the grouped null-space compensation payloads of ``ns_mode == 2`` checkpoints (the
        ``gate_ns`` / ``up_ns`` / ``down_ns`` entries of the reference's payload cache,
        modeling_olmoe.py:950-975; built by ``build_grouped_ns_compensation_payload``).  With any of
        them the layer's launch sequence gains the products of the pairs (``tris_moe_layer_forward_extras``)."""
        from .ns_compensation import ns_payload_max_rank

        self.ns_payloads = {n: p for n, p in (("gate", gate_ns), ("up", up_ns), ("down", down_ns))
                            if p is not None and ns_payload_max_rank(p) > 0}
        if self.ns_payloads and self.gate.weight.is_cuda:
            self._status_of(self.gate.weight.device)
        return self

    def backbone_rank(self, name: str) -> int:
        p = self.packed_backbones.get(name)
        return p.rows if p is not None else int(getattr(self, "shared_" + name).shape[0])

    def backbone_hidden(self, name: str, x: torch.Tensor, layout: int = 0) -> torch.Tensor:
        """``x . backbone^T`` (``compute_shared_hidden``) for the fp16 or the 4-bit form of a backbone."""
        scale = self.input_scales.get(name)
        if scale is not None:
            x = x * scale
        p = self.packed_backbones.get(name)
        if p is not None:
            return p(x, layout)
        return compute_shared_hidden(x, getattr(self, "shared_" + name), layout=layout)

    def _get_grouped_payload(self, cache_key: str) -> dict:
        if cache_key not in self._grouped_payload_cache:
            raise RuntimeError(f"trismoe_b200: grouped payload '{cache_key}' was not loaded")
        return self._grouped_payload_cache[cache_key]

    def layer_view(self) -> TrisMoeLayerView:
        views = [proj_view(self._get_grouped_payload(k)) for k in ("gate", "up", "down")]
        if self._layer_view is None or any(self._get_grouped_payload(k).get("_tris_layer_dirty") for k in ("gate", "up", "down")):
            v = TrisMoeLayerView()
            v.hidden_size, v.intermediate_size = self.hidden_size, self.intermediate_size
            v.num_experts, v.top_k, v.norm_topk_prob = self.num_experts, self.top_k, int(self.norm_topk_prob)
            v.router_weight = self.gate.weight.data_ptr()
            for name in ("gate", "up", "down"):
                p = self.packed_backbones.get(name)
                setattr(v, "shared_" + name, None if p is not None else getattr(self, "shared_" + name).data_ptr())
                setattr(v, "packed_" + name, None if p is None else C.addressof(p._view))
            v.gate, v.up, v.down = views
            for k in ("gate", "up", "down"):
                self._get_grouped_payload(k)["_tris_layer_dirty"] = False
            self._layer_view, self._expanded_view = v, None
        return self._layer_view

    def _expanded_layer_view(self, dev, names, own: Optional[list] = None) -> TrisMoeLayerView:
        """The layer view with the 4-bit backbones in ``names`` expanded into fp16 scratch (enqueued on
        the current stream): what large batches use, where the dense GEMM beats re-expanding nibbles for
        every pass over the rows.  The scratch is shared by all blocks of a model, or with ``own`` the call's
        own, kept in that list."""
        base = self.layer_view()
        if self._expanded_view is None:
            self._expanded_view = {}
        key = tuple(sorted(names))
        v = self._expanded_view.get(key) if own is None else None
        if v is None:
            v = TrisMoeLayerView()
            C.pointer(v)[0] = base
            if own is None:
                self._expanded_view[key] = v
        lib = _native.load()
        for name in key:
            p = self.packed_backbones[name]
            skey = (dev, name, p.rows, p.cols)
            scratch = TrisSparseMoeBlock._expand_scratch.get(skey) if own is None else None
            if scratch is None:
                scratch = torch.empty((p.rows, p.cols), dtype=torch.float16, device=dev)
                if own is None:
                    TrisSparseMoeBlock._expand_scratch[skey] = scratch
                else:
                    own.append(scratch)
            if getattr(p, "_g_idx", None) is None:
                g_idx = (torch.arange(p.cols, device=dev, dtype=torch.int32) // max(1, p.group_size)).clamp_(max=p.groups - 1)
                p._g_idx = g_idx.to(torch.int32).contiguous()
            with _native.on_device(dev):
                _native.check(lib.tris_packed4_dequantize(p.qweight.data_ptr(), p.qzeros.data_ptr(), p.scales.data_ptr(),
                                                          p._g_idx.data_ptr(), p.rows, p.cols, p.groups, scratch.data_ptr(),
                                                          _native.stream_of(dev)), "packed4_dequantize")
            setattr(v, "shared_" + name, scratch.data_ptr())
            setattr(v, "packed_" + name, None)
        return v

    def _layer_extras(self, dev) -> Optional[TrisMoeLayerExtras]:
        """Input scales and null-space pairs as the native layer takes them; None where it cannot: a router wider
        than its own, or scales and pairs of other sizes than the layer's, which the separate operators
        broadcast, skip or refuse."""
        from .ns_compensation import prepare_ns_payload

        H, I, E = self.hidden_size, self.intermediate_size, self.num_experts
        if E > 256 or self.top_k > 32:
            return None
        ex = TrisMoeLayerExtras()
        for i, (name, width, out) in enumerate((("gate", H, I), ("up", H, I), ("down", I, H))):
            scale = self.input_scales.get(name)
            if scale is not None:
                if scale.numel() != width or scale.device != dev:
                    return None
                ex.input_scale[i] = scale.data_ptr()
            if name in self.ns_payloads:
                p = prepare_ns_payload(self.ns_payloads[name], dev)
                c2, c1 = p["_tris_c2_view"], p["_tris_c1_view"]
                if (c2.k, c1.n, c2.num_experts) != (width, out, E):
                    return None
                ex.ns_c2[i], ex.ns_c1[i] = C.addressof(c2), C.addressof(c1)
        return ex

    def workspace(self, num_tokens: int, device, shared: Optional[TrisSharedExpert] = None) -> torch.Tensor:
        view = self.layer_view()
        width = 0 if shared is None else C.cast(shared.gate, C.POINTER(_native.TrisProjView))[0].out_features
        sized = self._workspace_for  # (view, shared expert's width, tokens) the buffer is known to hold: the size grows with the tokens
        if sized is not None and sized[0] is view and sized[1] == width and num_tokens <= sized[2] and self._workspace is not None and self._workspace.device == device:
            return self._workspace
        lib = _native.load()
        if shared is None:
            need = int(lib.tris_moe_layer_workspace_bytes(C.byref(view), int(num_tokens)))
        else:
            need = int(lib.tris_moe_layer_shared_workspace_bytes(C.byref(view), C.byref(shared), int(num_tokens)))
        if need == 0 and num_tokens > 0:
            raise RuntimeError("trismoe_b200: invalid layer view (workspace size query failed)")
        if self._workspace is None or self._workspace.numel() < need or self._workspace.device != device:
            if self._workspace is not None:
                self.raise_on_kernel_status()  # do not lose a report with the old buffer
            self._workspace = torch.empty((need,), dtype=torch.uint8, device=device)
            self._workspace[:16].zero_()  # count words and the sticky status word
        self._workspace_for = (view, width, int(num_tokens))
        return self._workspace

    def _extras_workspace(self, num_tokens: int, device, extras: TrisMoeLayerExtras) -> torch.Tensor:
        """Scratch of one call with input scales or null-space pairs: such blocks may be called from several threads and
        streams at once, as the separate operators may, so no buffer outlives the call."""
        need = int(_native.load().tris_moe_layer_extras_workspace_bytes(C.byref(self.layer_view()), C.byref(extras), int(num_tokens)))
        if need == 0:
            raise RuntimeError("trismoe_b200: invalid layer view (workspace size query failed)")
        return torch.empty((need,), dtype=torch.uint8, device=device)

    def _status_of(self, device) -> torch.Tensor:
        """Sticky status word of the kernels that do not report to a workspace of the block."""
        if self._status_word is None or self._status_word.device != device:
            self._status_word = torch.zeros((1,), dtype=torch.int32, device=device)
        return self._status_word

    def last_kernel_status(self, clear: bool = True) -> int:
        """Status word of every kernel :meth:`forward` launched since the last clear: 0, or 6
        (``TRIS_ERR_TIMEOUT``) when a bounded device-side wait ran out and a CTA skipped its stores.
        Synchronises the current stream; call it where the host waits for the GPU anyway (end of a
        decode step, before results are handed on)."""
        streamed = 0
        if self._status_word is not None:
            streamed = int(self._status_word.item())
            if clear and streamed:
                self._status_word.zero_()
        if self._workspace is None:
            return streamed
        lib = _native.load()
        dev = self._workspace.device
        word = C.c_int32(0)
        with _native.on_device(dev):
            _native.check(lib.tris_moe_layer_last_status(self._workspace.data_ptr(), int(bool(clear)),
                                                         _native.stream_of(dev), C.byref(word)),
                          "moe_layer_last_status")
        return int(word.value) or streamed

    def raise_on_kernel_status(self) -> None:
        """Raises ``RuntimeError`` if a kernel reported a time-out since the last check (the outputs
        of those calls are not trustworthy); the reference surfaces kernel failures as exceptions too."""
        status = self.last_kernel_status(clear=True)
        if status != 0:
            raise RuntimeError(f"trismoe_b200: a grouped kernel reported {_native.STATUS_NAMES.get(status, status)} "
                               "(TRIS_ERR_TIMEOUT: a bounded wait on a copy ran out; TRIS_ERR_WORKSPACE: a streamed batch activated "
                               "more experts than the staging manager has slots for; TRIS_ERR_CORRUPT: a streamed payload's column maps were changed "
                               "after its records were planned; output rows of that launch are stale)")

    def _require_rows(self, x: torch.Tensor, what: str) -> None:
        """The kernels take addresses: rows of another type or width would be misread or read out of range."""
        if x.dtype != torch.float16 or x.shape[-1] != self.hidden_size:
            raise RuntimeError(f"trismoe_b200 {what}: float16 hidden states of width {self.hidden_size} required, "
                               f"got {x.dtype} of width {x.shape[-1]}")

    # -- forward ---------------------------------------------------------------------------
    def forward(self, hidden_states: torch.Tensor, router_logits: Optional[torch.Tensor] = None):
        """Returns ``(final_hidden_states [B, S, H], router_logits [T, E])`` like
        ``OlmoeSparseMoeBlock.forward`` (modeling_olmoe.py:1046-1105).  ``router_logits``
        (fp32 ``[T, E]``) may be passed in to skip the router linear."""
        return self._forward(hidden_states, router_logits)

    def _forward(self, hidden_states: torch.Tensor, router_logits: Optional[torch.Tensor], shared: Optional[TrisSharedExpert] = None):
        """``shared``: a shared expert that joins the launch sequence (blocks without scales and pairs only)."""
        _native.require_cuda(hidden_states, "TrisSparseMoeBlock.forward")
        with_extras = bool(self.input_scales or self.ns_payloads)
        extras = self._layer_extras(hidden_states.device) if with_extras else None
        if not envflags.grouped_experts_enabled() or (with_extras and extras is None):
            # TRIS_GROUPED_EXPERTS=0, or scales and pairs that the native sequence does not take: operator by operator
            return self.forward_grouped_ops(hidden_states, router_logits)
        if hidden_states.dtype != torch.float16:
            raise RuntimeError(f"trismoe_b200: grouped expert kernels require float16 hidden states, got {hidden_states.dtype}")
        lib = _native.load()
        shape = hidden_states.shape
        if extras is None and hidden_states.is_contiguous() and shape[-1] == self.hidden_size:
            x, T = hidden_states, hidden_states.numel() // self.hidden_size  # as it is: the kernels take addresses
        else:
            x = hidden_states.reshape(-1, shape[-1]).contiguous()
            T = int(x.shape[0])
        dev = x.device
        y = torch.empty_like(x)
        returned = router_logits
        if extras is not None and router_logits is None:
            # such blocks route by fp16 logits and return them
            router_logits = returned = torch.nn.functional.linear(x, self.gate.weight)
        if router_logits is not None:
            logits = router_logits.reshape(T, self.num_experts).to(torch.float32).contiguous()
            logits_in, logits_out = logits.data_ptr(), None
        else:
            logits = torch.empty((T, self.num_experts), dtype=torch.float32, device=dev)
            logits_in, logits_out = None, logits.data_ptr()
        if T:
            self._require_rows(x, "forward")
            ws = self.workspace(T, dev, shared) if extras is None else self._extras_workspace(T, dev, extras)
            view = self._layer_view  # which the size query has just brought up to date
            own = None if extras is None else []
            if self.packed_backbones:  # gate and up see T rows, down T * top_k
                big = [n for n in self.packed_backbones
                       if (T * self.top_k if n == "down" else T) > self.PACKED_BACKBONE_MAX_ROWS]
                if "gate" in big or "up" in big:
                    big = sorted(set(big) | ({"gate", "up"} & set(self.packed_backbones)))
                if big:
                    view = self._expanded_layer_view(dev, big, own)
            with _native.on_device(dev):
                stream = _native.stream_of(dev)
                if shared is not None:
                    scratch = self._shared_scratch(lib, shared, T, dev)
                    st = lib.tris_moe_layer_forward_shared(C.byref(view), C.byref(shared), x.data_ptr(), logits_in, T, y.data_ptr(), logits_out,
                                                           ws.data_ptr(), ws.numel(), None if scratch is None else scratch.data_ptr(),
                                                           0 if scratch is None else scratch.numel(), stream)
                elif extras is None:
                    st = lib.tris_moe_layer_forward(C.byref(view), x.data_ptr(), logits_in, T, y.data_ptr(),
                                                    logits_out, ws.data_ptr(), ws.numel(), stream)
                else:
                    st = lib.tris_moe_layer_forward_extras_status(C.byref(view), C.byref(extras), x.data_ptr(), logits_in, T, y.data_ptr(),
                                                                  logits_out, ws.data_ptr(), ws.numel(), self._status_of(dev).data_ptr(), stream)
                _native.check(st, "moe_layer_forward")
        return y if x is hidden_states else y.reshape(shape), logits if extras is None else returned

    def forward_streaming(self, hidden_states: torch.Tensor, manager, block_index: int,
                          router_logits: Optional[torch.Tensor] = None):
        """Forward with the expert payloads paged in by a
        :class:`~.staging.GroupedQGmapCPUStagingManager` (the streaming mode of
        ``OlmoeModel.forward``, modeling_olmoe.py:1305-1339): the route is built first, the
        pager for gate/up/down starts on the side stream and overlaps the input-side backbone
        GEMM; the grouped kernels wait on its event.  Nothing synchronises with the host."""
        _native.require_cuda(hidden_states, "TrisSparseMoeBlock.forward_streaming")
        shape = hidden_states.shape
        x = hidden_states.reshape(-1, shape[-1]).contiguous()
        T, dev = int(x.shape[0]), x.device
        E, k, H, I = self.num_experts, self.top_k, self.hidden_size, self.intermediate_size
        R = T * k
        y = torch.empty_like(x)
        if T == 0:
            return y.reshape(shape), x.new_zeros((0, E), dtype=torch.float32)
        self._require_rows(x, "forward_streaming")
        lib = _native.load()
        r_gu, r_d = self.backbone_rank("gate"), self.backbone_rank("down")
        mode_gu, mode_d = (2 if r_gu % 32 == 0 else 0), (2 if r_d % 32 == 0 else 0)
        plain = lambda name: name not in self.packed_backbones and name not in self.input_scales
        if all(plain(name) for name in ("gate", "up", "down")):
            y, logits = self._forward_streaming_native(lib, x, y, manager, block_index, router_logits)
            return y.reshape(shape), logits
        with _native.on_device(dev):
            stream = _native.stream_of(dev)
            # one allocation for everything between the kernels; the host has 25 launches a layer to prepare
            sizes = [4 * R] * 6 + [4 * E, 4 * (E + 1), 4 * (E + 1), 16, 2 * T * r_gu, 2 * T * r_gu, 2 * R * I, 2 * R * r_d, 2 * R * H]
            offsets, total = [], 0
            for n in sizes:
                offsets.append(total)
                total += (n + 255) & ~255
            ws = torch.empty((total,), dtype=torch.uint8, device=dev)
            base = ws.data_ptr()
            sel, wts, perm, tok, slot, rof, ids, seg, prob, counts, hg, hu, mlp_ptr, hd, down = (base + o for o in offsets)
            projected = router_logits is None and plain("gate") and plain("up") and self.backbone_rank("up") == r_gu
            if router_logits is not None:
                logits = router_logits.reshape(T, E).to(torch.float32).contiguous()
            else:
                logits = torch.empty((T, E), dtype=torch.float32, device=dev)
                if projected:  # router and both input-side backbones in one launch
                    _native.check(lib.tris_input_projections(x.data_ptr(), T, H, self.shared_gate.data_ptr(), self.shared_up.data_ptr(), r_gu,
                                                             self.gate.weight.data_ptr(), E, hg, hu, mode_gu, logits.data_ptr(), stream),
                                  "input_projections")
                else:
                    _native.check(lib.tris_shared_hidden_forward(x.data_ptr(), None, T, None, H, self.gate.weight.data_ptr(), E,
                                                                 logits.data_ptr(), 1, stream), "router")
            _native.check(lib.tris_router_topk(logits.data_ptr(), T, E, k, int(self.norm_topk_prob), sel, wts, stream), "router_topk")
            _native.check(lib.tris_build_grouped_route(sel, T, k, E, 4, perm, tok, slot, rof, ids, seg, prob, counts, stream), "route")
            paged = manager.page_layer(block_index, {"expert_ids": ids, "segment_offsets": seg, "counts": counts, "experts": E,
                                                     "rows": R})  # side stream, starts now
            keep = []
            if not projected:
                keep = [self.backbone_hidden("gate", x, mode_gu), self.backbone_hidden("up", x, mode_gu)]
                hg, hu = keep[0].data_ptr(), keep[1].data_ptr()
            rv = _native.TrisRouteView()
            rv.expert_ids, rv.segment_offsets, rv.num_segments_dev = ids, seg, counts
            rv.num_segments, rv.num_rows, rv.max_rows_per_segment = min(E, R), R, T
            rv.row_gather, rv.status_dev, rv.flags = tok, self._status_of(dev).data_ptr(), (1 if mode_gu else 0)
            paged.wait("gate_up")  # down keeps paging under the gate/up kernel and the down backbone
            _native.check(lib.tris_grouped_pair_forward(C.byref(paged.views["gate"]), C.byref(paged.views["up"]), C.byref(rv), hg, hu, mlp_ptr,
                                                        None, 1, stream), "grouped_pair_forward")
            if plain("down"):
                _native.check(lib.tris_shared_hidden_forward(mlp_ptr, None, R, None, I, self.shared_down.data_ptr(), r_d, hd, mode_d, stream),
                              "down backbone")
            else:
                mlp = ws[offsets[12]: offsets[12] + 2 * R * I].view(torch.float16).view(R, I)
                keep.append(self.backbone_hidden("down", mlp, mode_d))
                hd = keep[-1].data_ptr()
            rv.row_gather, rv.flags = None, (1 if mode_d else 0)
            paged.wait("all")
            _native.check(lib.tris_grouped_forward(C.byref(paged.views["down"]), C.byref(rv), hd, down, stream), "grouped_forward")
            paged.release()
            _native.check(lib.tris_combine_routed(down, rof, wts, T, k, H, y.data_ptr(), stream), "combine")
        return y.reshape(shape), logits

    def _forward_streaming_native(self, lib, x, y, manager, block_index, router_logits):
        """The same as one native call over both streams (``tris_moe_layer_forward_paged``)."""
        T, E, dev = int(x.shape[0]), self.num_experts, x.device
        view = self.layer_view()
        if router_logits is not None:
            logits = router_logits.reshape(T, E).to(torch.float32).contiguous()
            logits_in, logits_out = logits.data_ptr(), None
        else:
            logits = torch.empty((T, E), dtype=torch.float32, device=dev)
            logits_in, logits_out = None, logits.data_ptr()
        with _native.on_device(dev):
            need = int(lib.tris_moe_layer_workspace_bytes(C.byref(view), T))
            if need == 0:
                raise RuntimeError("trismoe_b200: invalid layer view (workspace size query failed)")
            ws = torch.empty((need,), dtype=torch.uint8, device=dev)
            status = self._status_of(dev).data_ptr()
            with manager.native_layer(block_index, T * self.top_k, E) as paged:
                _native.check(lib.tris_moe_layer_forward_paged(C.byref(view), C.byref(paged), x.data_ptr(), logits_in, T, y.data_ptr(), logits_out,
                                                               ws.data_ptr(), need, status, _native.stream_of(dev)), "moe_layer_forward_paged")
        return y, logits

    def forward_grouped_ops(self, hidden_states: torch.Tensor, router_logits: Optional[torch.Tensor] = None):
        """Same result as :meth:`forward`, composed from the reference-named operators in
        the order of ``_forward_grouped`` (modeling_olmoe.py:916-1044); torch is used only
        for the glue the reference also does in torch (softmax/top-k, gathers, act*mul,
        index_add_)."""
        shape = hidden_states.shape
        x = hidden_states.reshape(-1, shape[-1])
        if router_logits is None:
            router_logits = torch.nn.functional.linear(x, self.gate.weight)
        if x.shape[0] == 0:
            return x.new_zeros(shape), router_logits
        routing = torch.softmax(router_logits, dim=1, dtype=torch.float)
        routing, selected = torch.topk(routing, self.top_k, dim=-1)
        if self.norm_topk_prob:
            routing = routing / routing.sum(dim=-1, keepdim=True)
        routing = routing.to(x.dtype)
        route = build_grouped_route(selected, self.num_experts)
        tok, slots = route["grouped_token_indices"], route["grouped_slots"]
        x_grouped = x.index_select(0, tok)
        grouped_routing = routing[tok, slots].unsqueeze(-1)
        gate_hidden = self.backbone_hidden("gate", x).index_select(0, tok)
        up_hidden = self.backbone_hidden("up", x).index_select(0, tok)
        gate_out, up_out = run_grouped_structured_expert_pair_forward(
            self._get_grouped_payload("gate"), self._get_grouped_payload("up"), gate_hidden, up_hidden, x_grouped, route,
            ns_payload_a=self.ns_payloads.get("gate"), ns_payload_b=self.ns_payloads.get("up"))
        mlp = torch.nn.functional.silu(gate_out) * up_out
        down_hidden = self.backbone_hidden("down", mlp)
        down_out = run_grouped_structured_expert_forward(self._get_grouped_payload("down"), down_hidden, mlp, route,
                                                         ns_payload=self.ns_payloads.get("down"))
        # weighted sum of every token's k expert rows, taken in slot order (the reference scatters them with
        # index_add_, whose atomic order varies from run to run; this is the same sum, reproducible)
        weighted = (down_out * grouped_routing).to(x.dtype)
        rows_of_token = route["_row_of_flat"].to(torch.long)
        final = weighted.index_select(0, rows_of_token).view(x.shape[0], self.top_k, x.shape[1]).float().sum(dim=1).to(x.dtype)
        return final.reshape(shape), router_logits


class TrisQwen2SparseMoeBlock(TrisSparseMoeBlock):
    """``Qwen2MoeSparseMoeBlock`` of the reference (modeling_qwen2_moe.py:249-822): the routed experts
    of :class:`TrisSparseMoeBlock` plus one always-on shared expert - a dense gate/up/down MLP of
    ordinary compact3 linears whose output is scaled by ``sigmoid(shared_expert_gate(x))`` and added
    (modeling_qwen2_moe.py:815-818).  The shared expert's gate and up run as one dual launch with
    SiLU*mul fused (``run_compact3_shared_expert_gate_up_forward``, modeling_qwen2_moe.py:117-123)."""

    def __init__(self, hidden_size: int, intermediate_size: int, num_experts: int, num_experts_per_tok: int,
                 norm_topk_prob: bool = False):
        super().__init__(hidden_size, intermediate_size, num_experts, num_experts_per_tok, norm_topk_prob)
        self.shared_expert_gate = nn.Linear(self.hidden_size, 1, bias=False, dtype=torch.float16)
        self.shared_expert = None  # (gate, up, down) Compact3Linear

    def load_shared_expert(self, gate_proj, up_proj, down_proj, shared_expert_gate_weight: torch.Tensor, device=None):
        """``gate_proj`` / ``up_proj`` / ``down_proj``: :class:`~.compact3_linear.Compact3Linear` modules or the
        per-module compact3 payload dicts they are built from; ``shared_expert_gate_weight``: ``[1, hidden]``."""
        from .compact3_linear import Compact3Linear

        dev = torch.device(device) if device is not None else self.gate.weight.device
        mods = [m if isinstance(m, Compact3Linear) else Compact3Linear(m, device=dev) for m in (gate_proj, up_proj, down_proj)]
        self.shared_expert = tuple(mods)
        self.shared_expert_gate.weight = nn.Parameter(shared_expert_gate_weight.reshape(1, self.hidden_size).to(dev, torch.float16).contiguous(),
                                                      requires_grad=False)
        return self

    def _shared_view(self, hidden_states: torch.Tensor) -> Optional[TrisSharedExpert]:
        """The shared expert as the native layer takes it; None where the separate operators have to run: planes without tile records,
        scales, other sizes, types or places, gradients, hooks on the down projection."""
        from .compact3_linear import Compact3Linear

        mods, w, H = self.shared_expert, self.shared_expert_gate.weight, self.hidden_size
        if self.input_scales or self.ns_payloads or not envflags.grouped_experts_enabled() or not all(type(m) is Compact3Linear for m in mods):
            return None
        gate, up, down = mods
        hooks = torch.nn.modules.module._has_any_global_hook() or down._forward_hooks or down._forward_pre_hooks
        if (hooks or any(m.input_scale is not None or m.payload.get("_tris_tile_records") is None for m in mods)
                or (gate.in_features, up.in_features, up.out_features, down.in_features, down.out_features)
                != (H, H, gate.out_features, gate.out_features, H)):
            return None
        dev = hidden_states.device
        if (hidden_states.dtype != torch.float16 or w.dtype != torch.float16 or w.shape != (1, H) or not w.is_contiguous() or H % 8
                or hidden_states.shape[-1] != H or dev.type != "cuda" or w.device != dev
                or any(m.payload["qweight1"].device != dev for m in mods)
                or (torch.is_grad_enabled() and (w.requires_grad or hidden_states.requires_grad))):
            return None
        return TrisSharedExpert(*(C.addressof(proj_view(m.payload)) for m in mods), w.data_ptr())

    @staticmethod
    def _shared_scratch(lib, shared: TrisSharedExpert, rows: int, device) -> Optional[torch.Tensor]:
        """Scratch of one call for the shared expert's two launches, as the separate operators take it (a block's own buffer would hold on to
        up to 256 MB of it)."""
        if rows <= 32:
            return None
        need = max(int(lib.tris_linear_workspace_bytes(C.cast(p, C.POINTER(_native.TrisProjView)), n, rows)) for p, n in ((shared.gate, 2), (shared.down, 1)))
        return torch.empty((need,), dtype=torch.uint8, device=device) if need else None

    def forward(self, hidden_states: torch.Tensor, router_logits: Optional[torch.Tensor] = None):
        from .compact3_linear import run_compact3_gate_up_forward

        if self.shared_expert is None:
            raise RuntimeError("trismoe_b200: the shared expert was not loaded (load_shared_expert)")
        view = self._shared_view(hidden_states)
        if view is not None:
            return self._forward(hidden_states, router_logits, view)
        routed, logits = super().forward(hidden_states, router_logits)
        gate_proj, up_proj, down_proj = self.shared_expert
        mlp = run_compact3_gate_up_forward(gate_proj, up_proj, hidden_states, fuse_silu_mul=True)
        shared = down_proj(mlp)
        if shared is None:
            raise RuntimeError("trismoe_b200: shared expert kernels returned no result")
        w = self.shared_expert_gate.weight
        dev, f16 = routed.device, torch.float16
        native = (w.dtype == hidden_states.dtype == routed.dtype == shared.dtype == f16 and w.device == dev and hidden_states.device == dev
                  and w.shape == (1, self.hidden_size) and routed.is_contiguous() and w.is_contiguous()
                  and not (torch.is_grad_enabled() and (w.requires_grad or hidden_states.requires_grad)))
        if not native:  # torch's own checks of the gate's size and place, and its gradients
            return routed + torch.sigmoid(torch.nn.functional.linear(hidden_states, w)) * shared, logits
        x, shared = hidden_states.contiguous(), shared.contiguous()
        T = routed.numel() // self.hidden_size
        with _native.on_device(routed.device):
            _native.check(_native.load().tris_shared_expert_add(x.data_ptr(), w.data_ptr(), routed.data_ptr(), shared.data_ptr(), T, self.hidden_size,
                                                                routed.data_ptr(), _native.stream_of(routed.device)),
                          "shared_expert_add")
        return routed, logits
