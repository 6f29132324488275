"""Timed workloads of the framework: what a serving or evaluation program has it do, through its
public entry points.

``listed()`` names the workloads, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes what a
program holds before the call (weights, payloads, managers, captured graphs, inputs), ``run`` is one
pass, ``work`` what a pass cannot do without and ``tolerance`` how far two correct implementations
may be apart.  All data is synthetic and made on the GPU from the seed: sign planes Bernoulli(0.5),
salient columns and grouping bits Bernoulli(0.1), row scales |N(0, 0.02)|, column scales around 1,
backbones N(0, 0.02), activations N(0, 1) with 1 % of the channels scaled by 20.
"""
import math

import torch

import trismoe_b200 as tm
from trismoe_b200.staging import GroupedQGmapCPUStagingManager

GROUP = 128
P_SALIENT = P_GMAP = 0.1
# hidden, expert intermediate, experts, top-k: the layer shapes of the benchmark and the tests
MODELS = {"olmoe": (2048, 1024, 64, 8), "mixtral": (4096, 14336, 8, 2), "qwen35": (2048, 512, 256, 8)}
# hidden, q width, k/v width of the attention projections around those layers
ATTENTION = {"olmoe": (2048, 2048, 2048), "mixtral": (4096, 4096, 1024), "qwen35": (2048, 4096, 512)}


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def _case(kind, model, tokens, **more):
    return dict({"kind": kind, "model": model, "tokens": tokens, "rank": 256}, **more)


def listed():
    cases = {
        # one token at a time, the interactive case: a captured decode step over several layers
        "decode 1 graph": _case("block", "olmoe", 1, layers=4, graph=True, backbone="fp16"),
        # a small batch called eagerly, layer by layer, as a model's forward does without graphs
        "decode 8 eager": _case("block", "olmoe", 8, layers=1, graph=False, backbone="fp16"),
        # the benchmark's headline: a decode batch of 128 through distinct layers
        "decode 128 graph": _case("block", "olmoe", 128, layers=4, graph=True, backbone="fp16"),
        # few large experts at a medium batch
        "mixtral decode 64": _case("block", "mixtral", 64, layers=1, graph=False, backbone="fp16"),
        # backbones as real checkpoints store them (4 bits), decode batch
        "decode 16 packed4": _case("block", "olmoe", 16, layers=1, graph=False, backbone="packed4"),
        # prompts: an odd length, a long one, and a long one through the large experts
        "prefill 509": _case("block", "olmoe", 509, layers=1, graph=False, backbone="fp16"),
        "prefill 2048": _case("block", "olmoe", 2048, layers=1, graph=False, backbone="fp16"),
        "mixtral prefill 2048": _case("block", "mixtral", 2048, layers=1, graph=False, backbone="fp16"),
        # many small experts plus the always-on shared expert
        "shared expert 16": _case("shared", "qwen35", 16),
        # checkpoints with a null-space pair per expert: the reference-named operators one by one
        "null-space 37": _case("nullspace", "olmoe", 37),
        # attention projections of a quantised checkpoint (grouped-query widths)
        "qkv 512": _case("qkv", "mixtral", 512),
        # experts in pinned host memory, paged per layer
        "streaming 16": _case("streaming", "qwen35", 16, layers=2, mode="bitmap"),
    }
    return [dict(c, name=name) for name, c in cases.items()]


def _log_int(rng, low, high):
    return min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(["block"] * 6 + ["shared", "nullspace", "qkv", "streaming"])
    model = rng.choice(list(MODELS))
    if kind == "block":
        tokens = _log_int(rng, 1, 2048)
        decode = tokens <= 128
        return _case(kind, model, tokens, layers=rng.randint(1, 4) if decode and model != "mixtral" else 1,
                     graph=decode and rng.random() < 0.5, backbone="packed4" if rng.random() < 0.25 else "fp16",
                     rank=rng.choice([128, 256, 256, 256, 320]))
    if kind == "shared":
        return _case(kind, "qwen35", _log_int(rng, 1, 1024))
    if kind == "nullspace":
        return _case(kind, "olmoe", _log_int(rng, 1, 512))
    if kind == "qkv":
        return _case(kind, model, _log_int(rng, 1, 512))
    return _case(kind, rng.choice(["olmoe", "qwen35"]), _log_int(rng, 1, 32), layers=rng.randint(1, 3),
                 mode=rng.choice(["bitmap", "payload"]))


# ---------------------------------------------------------------------------------------
# synthetic data on the GPU
# ---------------------------------------------------------------------------------------
def _pack_words(bits, dim):
    """Packs 32 entries along ``dim`` into int32 words, entry j at bit j."""
    shape = [1] * bits.dim()
    shape[dim] = 32
    weight = (torch.ones(32, dtype=torch.int64, device=bits.device) << torch.arange(32, device=bits.device)).to(torch.int32)
    return (bits.to(torch.int32) * weight.view(shape)).sum(dim=dim, dtype=torch.int32)


def _block_gr(bits):
    """Block Golomb-Rice streams of grouping bits ``[E, pr, 32, O]`` (blocks of two packed rows by 64
    outputs, in (row, output, bit) order): words ``[E, longest]``, offsets and meta."""
    E, pr, _, O = bits.shape
    nkb, nob = -(-pr // 2), -(-O // 64)
    bits = torch.nn.functional.pad(bits, (0, nob * 64 - O, 0, 0, 0, nkb * 2 - pr))
    flat = bits.view(E, nkb, 2, 32, nob, 64).permute(0, 1, 4, 2, 5, 3).reshape(E * nkb * nob, 4096)
    blk, pos = flat.nonzero(as_tuple=True)
    first = torch.ones_like(blk, dtype=torch.bool)
    first[1:] = blk[1:] != blk[:-1]
    run = pos.clone()
    run[1:] = torch.where(first[1:], pos[1:], pos[1:] - pos[:-1] - 1)
    count = flat.sum(dim=1)
    cost = torch.stack([torch.zeros_like(count).index_add_(0, blk, run >> k) + count * (1 + k) for k in range(8)])
    best = (cost * 8 + torch.arange(8, device=bits.device)[:, None]).min(dim=0).values  # fewest bits, then lowest k
    k_of, words_of = best % 8, (best // 8 + 31) // 32
    assert int(words_of.max()) < 128
    offsets = torch.nn.functional.pad(words_of.view(E, -1).cumsum(1), (1, 0))
    longest = int(offsets[:, -1].max())
    base = (offsets[:, :-1] + longest * torch.arange(E, device=bits.device)[:, None]).reshape(-1) * 32
    k = k_of[blk]
    length = (run >> k) + 1 + k
    start = length.cumsum(0) - length
    stop = start + (run >> k) + base[blk] - start[first].repeat_interleave(count[count > 0])  # where the 1 of the unary part goes
    stream = torch.zeros((E * longest * 32,), dtype=torch.bool, device=bits.device)
    stream[stop] = True
    for j in range(7):
        stream[stop[(k > j) & ((run >> j) & 1).bool()] + 1 + j] = True
    return (_pack_words(stream.view(E, longest, 32), 2), offsets.to(torch.int32), (k_of | (count << 8)).to(torch.int32).view(E, -1))


def _projection(g, E, O, rank, block_gr=True):
    """E-stacked compact3 payload with random planes and scales."""
    dev, pr, G = g.device, -(-rank // 32), -(-rank // GROUP)
    rand = lambda *s: torch.rand(s, generator=g, device=dev)
    words = lambda *s: torch.randint(-2**31, 2**31, s, generator=g, device=dev, dtype=torch.int64).to(torch.int32)
    half = lambda mean, std, *s: (mean + std * torch.randn(s, generator=g, device=dev)).half()
    join = lambda *h: sum((t.view(torch.int16).to(torch.int64) & 0xFFFF) << (16 * i) for i, t in enumerate(h))
    valid = torch.arange(pr * 32, device=dev) < rank
    salient = (rand(E, pr * 32) < P_SALIENT) & valid
    rest = ~salient & valid
    prefix = lambda m: torch.nn.functional.pad(m.view(E, pr, 32).sum(2).cumsum(1), (1, 0)).to(torch.int32)
    count = salient.sum(1)
    sal_rows = max(1, -(-int(count.max()) // 32))
    in_slot = torch.arange(sal_rows * 32, device=dev)[None] < count[:, None]
    bits = (rand(E, pr, 32, O) < P_GMAP) & rest.view(E, pr, 32, 1)
    payload = {
        "is_compact3": True,
        "qweight1": words(E, pr, O) & _pack_words(valid.view(pr, 32), 1)[:, None],
        "qweight2_sparse": words(E, sal_rows, O) & _pack_words(in_slot.view(E, sal_rows, 32), 2)[:, :, None],
        "qweight2_sparse_prefix": prefix(salient),
        "q_gmap_sparse_prefix": prefix(rest),
        "c_map": _pack_words(salient.view(E, pr, 32), 2),
        "g_idx": (torch.arange(rank, device=dev, dtype=torch.int32) // GROUP).expand(E, rank).contiguous(),
        "col_pack3": join(*(half(1.0, 0.1, E, rank) for _ in range(4))),
        "row_pack3": join(*(half(0.0, std, E, O, G).abs() for std in (0.02, 0.01, 0.04, 0.02))),
        "output_scale": torch.ones((E, O), dtype=torch.float16, device=dev), "has_output_scale": False,
        "bias": None, "has_bias": False, "compact3_use_block_gr": block_gr,
    }
    if block_gr:
        payload["q_gmap_sparse"] = torch.zeros((E, 0, O), dtype=torch.int32, device=dev)
        payload["q_gmap_gr_words"], payload["q_gmap_gr_offsets"], payload["q_gmap_gr_meta"] = _block_gr(bits)
    else:
        order = torch.argsort((~rest).to(torch.int8), dim=1, stable=True)
        rows = -(-int(rest.sum(1).max()) // 32)
        packed = bits.view(E, pr * 32, O).gather(1, order[:, : rows * 32, None].expand(-1, -1, O)) if rows * 32 <= pr * 32 else bits
        payload["q_gmap_sparse"] = _pack_words(packed.reshape(E, rows, 32, O), 2)
        for key in ("q_gmap_gr_words", "q_gmap_gr_offsets", "q_gmap_gr_meta"):
            payload[key] = torch.empty((0, 0), dtype=torch.int32, device=dev)
    return payload


def _packed4(g, rows, cols, scale):
    """Random 4-bit packed matrix with groups of 128 input columns."""
    groups = max(1, -(-cols // GROUP))
    words = lambda *s: torch.randint(-2**31, 2**31, s, generator=g, device=g.device, dtype=torch.int64).to(torch.int32)
    return {"qweight": words(-(-cols // 8), rows), "qzeros": words(groups, -(-rows // 8)),
            "scales": (scale * torch.randn((groups, rows), generator=g, device=g.device)).abs().half(),
            "g_idx": torch.arange(cols, device=g.device, dtype=torch.int32) // GROUP, "rows": rows, "cols": cols}


def _activations(g, tokens, width):
    x = torch.randn((tokens, width), generator=g, device=g.device)
    x[:, torch.randperm(width, generator=g, device=g.device)[: max(1, width // 100)]] *= 20.0
    return x.half()


def _block(g, case, cls=tm.TrisSparseMoeBlock, block_gr=True):
    hidden, inter, experts, top_k = MODELS[case["model"]]
    rank = case["rank"]
    normal = lambda std, *s: (std * torch.randn(s, generator=g, device=g.device)).half()
    if case.get("backbone") == "packed4":
        backbone = lambda width: _packed4(g, rank, width, 0.004)
    else:
        backbone = lambda width: normal(0.02, rank, width)
    blk = cls(hidden, inter, experts, top_k, True)
    blk.load_grouped_payloads(_projection(g, experts, inter, rank, block_gr), _projection(g, experts, inter, rank, block_gr),
                              _projection(g, experts, hidden, rank, block_gr), backbone(hidden), backbone(hidden), backbone(inter),
                              normal(hidden ** -0.5, experts, hidden), device=g.device)
    return blk


def _nullspace(g, experts, width, out):
    """Compensation payload: every expert a 4-bit pair of null-space rank 32 or 64."""
    ranks = [32 * (1 + int(v)) for v in torch.randint(0, 2, (experts,), generator=g, device=g.device).tolist()]
    pairs = [{"c2": _packed4(g, r, width, 0.1 * width ** -0.5), "c1": _packed4(g, out, r, 0.1 * r ** -0.5)} for r in ranks]
    return tm.build_grouped_ns_compensation_payload(pairs, g.device, torch.float16, width, out)


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    state = {"kind": kind}
    hidden, inter, experts, _ = MODELS[case["model"]]
    if kind in ("block", "streaming"):
        state["blocks"] = [_block(g, case, block_gr=case.get("mode") != "bitmap") for _ in range(case["layers"])]
    elif kind == "shared":
        blk = _block(g, case, cls=tm.TrisQwen2SparseMoeBlock)
        blk.load_shared_expert(_projection(g, 1, inter, hidden), _projection(g, 1, inter, hidden), _projection(g, 1, hidden, inter),
                               (hidden ** -0.5 * torch.randn((1, hidden), generator=g, device=g.device)).half())
        state["blocks"] = [blk]
    elif kind == "nullspace":
        blk = _block(g, case)
        blk.load_ns_compensation_payloads(_nullspace(g, experts, hidden, inter), _nullspace(g, experts, hidden, inter),
                                          _nullspace(g, experts, inter, hidden))
        state["blocks"] = [blk]
    elif kind == "qkv":
        hidden, q, kv = ATTENTION[case["model"]]
        state["linears"] = [tm.Compact3Linear(_projection(g, 1, width, hidden)) for width in (q, kv, kv)]
    state["x"] = _activations(g, case["tokens"], hidden).view(1, case["tokens"], hidden)
    if kind == "streaming":
        state["manager"] = GroupedQGmapCPUStagingManager(state["blocks"], mode=case["mode"])
        state["manager"].collect_timings = False
        state["manager"].initialize()
    if case.get("graph"):  # a decode step captured once, replayed for every token
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _forward(state)
        torch.cuda.current_stream().wait_stream(side)
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["out"] = _forward(state)
    return state


def _forward(state):
    if state["kind"] == "qkv":
        return tm.run_compact3_qkv_forward(*state["linears"], state["x"])
    if state["kind"] == "streaming":
        return [blk.forward_streaming(state["x"], state["manager"], i) for i, blk in enumerate(state["blocks"])]
    return [blk(state["x"]) for blk in state["blocks"]]


def run(state):
    with torch.no_grad():
        if "graph" in state:
            state["graph"].replay()
            return state["out"]
        return _forward(state)


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _expert_bytes(out, rank):
    """Compressed bytes of one expert matrix: signs, salient signs, Golomb-Rice coded grouping bits with
    their offsets and meta, column tables, scales."""
    weights = out * rank
    blocks = -(-rank // 64) * -(-out // 64)
    return weights / 8 + weights * P_SALIENT / 8 + weights * 0.9 * P_GMAP * 4.8 / 8 + 8 * blocks + 9 * rank + 8 * out * -(-rank // GROUP)


def _moe_work(case, streamed=False):
    hidden, inter, experts, k = MODELS[case["model"]]
    tokens, rank = case["tokens"], case["rank"]
    active = experts * (1.0 - (1.0 - k / experts) ** tokens)
    per_value = 4 / 8 + 2.5 / GROUP if case.get("backbone") == "packed4" else 2.0
    size = active * (2 * _expert_bytes(inter, rank) + _expert_bytes(hidden, rank))
    size += per_value * rank * (2 * hidden + inter) + 2 * experts * hidden + 4 * tokens * hidden + 4 * tokens * experts
    flops = 2.0 * tokens * hidden * (2 * rank + experts) + 2.0 * tokens * k * rank * (2 * inter + inter + hidden)
    return size, flops


def work(case):
    kind, tokens = case["kind"], case["tokens"]
    if kind == "qkv":
        hidden, q, kv = ATTENTION[case["model"]]
        size = _expert_bytes(q, hidden) + 2 * _expert_bytes(kv, hidden) + 2.0 * tokens * (hidden + q + 2 * kv)
        return {"bytes": size, "flops": 2.0 * tokens * hidden * (q + 2 * kv)}
    size, flops = _moe_work(case)
    hidden, inter, experts, k = MODELS[case["model"]]
    if kind == "shared":
        size += 2 * _expert_bytes(inter, hidden) + _expert_bytes(hidden, inter) + 2 * hidden
        flops += 6.0 * tokens * hidden * inter
    if kind == "nullspace":
        pairs = 48 * (3 * hidden + 3 * inter)  # values of the three pairs of an expert at the mean rank
        size += experts * (1.0 - (1.0 - k / experts) ** tokens) * pairs * (4 / 8 + 2.5 / GROUP)
        flops += 2.0 * tokens * k * pairs
    layers = case.get("layers", 1)
    return {"bytes": size * layers, "flops": flops * layers}


def tolerance(case):
    # fp16 weights and activations, fp32 sums, four roundings to fp16 (2^-11 each) between input and
    # output.  `max`: where two of a token's router logits are equal to the last bits of an fp32 sum, another
    # order of that sum picks the other expert for the smallest of the k weights.
    return {"rel": 3e-3, "max": 0.5}
