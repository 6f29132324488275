"""The tile-record kernels, the 4-bit GEMM and the backbone GEMM at the edges of their tiles and of the rules
that choose between their variants.  Weights are fp16 values known exactly (the dequantised matrix), so the
bound of an output is that of its sum: fp32 accumulation of products of fp16 values, then one rounding to fp16."""
import numpy as np
import pytest
import torch

from helpers import kernels_of, to_numpy_payload

pytestmark = pytest.mark.gpu


def _bound(w, h):
    """|error| of fp16(sum of w * h over k terms): half an fp16 ulp of the result (or of the smallest
    normal), plus k additions of relative error 2^-22 (truncating fp32 adds) of the sum of magnitudes."""
    ref = h.double() @ w.double().T
    mag = h.double().abs() @ w.double().abs().T
    acc = h.shape[1] * 2.0 ** -22 * mag
    return ref, acc, acc * (1 + 2.0 ** -10) + ref.abs() * 2.0 ** -11 + 2.0 ** -25


def _assert_within(got, ref, bound):
    worst = ((got.double() - ref).abs() / bound).max().item()
    assert worst <= 1.0, worst


def _payload(tm, E, O, rank, group, seed, **more):
    from trismoe_b200 import synth

    rng = np.random.default_rng(seed)
    p = synth.pack_projection(synth.raw_projection(rng, E, O, rank, group_size=group, **more))
    return tm.prepare_grouped_payload(p, "cuda")


# Few experts on the tiled kernel, in passes of 64 and of 128 rows: more units than the decode kernel's passes are taken for.
SHORT, UNEVEN = [130] + [43] * 31, [150, 50, 60, 65, 80, 55, 70, 30] * 4

# (outputs, rank, scale group, rows per expert): decode kernel with 8 / 4 / 2 / 1 warps per 32 outputs and 8 to 32
# rows per pass, a segment of several passes, more columns than one stage holds; tiled kernel with 64- and
# 128-row tiles (the last seven lines: one to five column chunks, two passes and more), ragged last tile; kernel for long
# segments; one to several tiles per CTA.
GROUPED = [
    (96, 256, 32, [1, 0, 8, 3]),
    (97, 264, 128, [16, 9, 16]),
    (33, 1040, 64, [2, 5]),
    (64, 64, 32, [24, 17, 0, 23]),
    (160, 80, 32, [70, 1, 1, 1, 1, 1, 1, 1]),
    (1040, 64, 64, [25 + i % 8 for i in range(40)]),
    (1031, 72, 128, [i % 5 for i in range(50)]),
    (2080, 320, 128, [1 + i % 3 for i in range(34)]),
    (2048, 44, 32, [1] * 34),
    (129, 136, 32, [33, 64, 65, 1]),
    (256, 520, 128, [129, 0, 257, 100]),
    (90, 44, 32, [300, 40]),
    (1040, 320, 128, [33 + i % 32 for i in range(40)]),  # several tiles per CTA on 3 and 4 staged chunks, several passes
    (1040, 512, 128, [70] + [33 + i % 32 for i in range(39)]),
    (1040, 300, 128, [70 + 9 * i for i in range(24)]),
    (33, 264, 128, [128, 40]),  # decode kernel, several CTAs to a segment's passes: up to 128 rows, few experts
    (1031, 72, 32, [97, 33, 64]),
    (64, 1040, 64, [65, 0, 31]),
    (2048, 256, 128, [100]),
    (520, 72, 32, SHORT),
    (520, 192, 64, SHORT),
    (520, 320, 128, SHORT[:-1]),
    (416, 128, 64, UNEVEN),
    (416, 192, 32, UNEVEN),
    (416, 320, 128, UNEVEN[:-1]),
    (416, 520, 64, UNEVEN[:-1]),
]


@pytest.mark.parametrize("O,rank,group,lengths", GROUPED)
def test_grouped_kernels_at_tile_edges(lib, O, rank, group, lengths):
    import trismoe_b200 as tm

    E, R = len(lengths), sum(lengths)
    pa, pb = _payload(tm, E, O, rank, group, O + rank), _payload(tm, E, O, rank, group, O + rank + 1)
    wa, wb = tm.dequantize_grouped_payload(pa), tm.dequantize_grouped_payload(pb)
    g = torch.Generator().manual_seed(R)
    ha, hb = ((0.5 * torch.randn((R, rank), generator=g)).half().cuda() for _ in range(2))
    one = tm.run_grouped_structured_expert_forward(pa, ha, None, lengths)
    sa, sb = tm.run_grouped_structured_expert_pair_forward(pa, pb, ha, hb, None, lengths)
    mlp, _ = tm.run_grouped_structured_expert_pair_forward(pa, pb, ha, hb, None, lengths, fuse_silu_mul=True)
    row = 0
    for e, n in enumerate(lengths):
        if n == 0:
            continue
        rows = slice(row, row + n)
        row += n
        ra, ea, ba = _bound(wa[e], ha[rows])
        rb, eb, bb = _bound(wb[e], hb[rows])
        _assert_within(one[rows], ra, ba)
        _assert_within(sa[rows], ra, ba)
        _assert_within(sb[rows], rb, bb)
        silu = ra * torch.sigmoid(ra)
        want = silu * rb  # |silu'| < 1.1; exponential, division and two products in fp32
        err = 1.1 * ea * rb.abs() + silu.abs() * eb + 1.1 * ea * eb + want.abs() * (2.0 ** -11 + 2.0 ** -19) + 2.0 ** -25
        _assert_within(mlp[rows], want, err)


@pytest.mark.parametrize("O,rank,group,lengths", GROUPED)
def test_grouped_kernels_give_every_single_weight(lib, O, rank, group, lengths):
    """Rows that are one at one column and zero elsewhere: an output is a single weight, exactly, so one lost or misplaced
    column or salient term shows whatever the size of a sum.  Every segment sees every column."""
    import trismoe_b200 as tm

    E = len(lengths)
    pa, pb = _payload(tm, E, O, rank, group, O + rank), _payload(tm, E, O, rank, group, O + rank + 1)
    wa, wb = tm.dequantize_grouped_payload(pa), tm.dequantize_grouped_payload(pb)
    expert = torch.repeat_interleave(torch.arange(E), torch.tensor(lengths)).cuda()
    place = torch.cat([torch.arange(n) for n in lengths]).cuda()
    route = tm.qlinear_grouped._coerce_grouped_route(lengths, "cuda")
    for c in range(0, rank, min(n for n in lengths if n)):
        ca, cb = (place + c) % rank, (place + c + 7) % rank
        ha, hb = (torch.nn.functional.one_hot(col, rank).half() for col in (ca, cb))
        assert torch.equal(tm.run_grouped_structured_expert_forward(pa, ha, None, route), wa[expert, :, ca])
        sa, sb = tm.run_grouped_structured_expert_pair_forward(pa, pb, ha, hb, None, route)
        assert torch.equal(sa, wa[expert, :, ca]) and torch.equal(sb, wb[expert, :, cb])


# Which kernel a call reaches, single projection and gate/up pair with SiLU: the rules by columns, experts and typical rows (mean and
# two standard deviations), either side of each line.
DECODE, TILED64, TILED128, WIDE_KERNEL = "grouped_decode_kernel<", "grouped_tiled_kernel<64,", "grouped_tiled_kernel<128,", "grouped_wide_kernel<"
REACHES = [
    (136, 128, [20] * 40, DECODE, DECODE),
    (264, 128, [130] + [35] * 39, DECODE, DECODE),     # 50 typical rows, all passes at once
    (520, 72, SHORT, TILED64, TILED64),                # 60
    (520, 192, SHORT, TILED64, TILED64),
    (520, 320, SHORT, WIDE_KERNEL, WIDE_KERNEL),
    (520, 320, SHORT[:-1], TILED64, TILED64),          # one expert less
    (416, 128, UNEVEN, TILED128, TILED128),            # 89
    (416, 192, UNEVEN, TILED128, TILED128),
    (416, 320, UNEVEN[:-1], TILED128, TILED128),
    (416, 520, UNEVEN[:-1], TILED128, TILED128),
    (1500, 128, [170] + [80] * 7, TILED128, TILED128), # 111, few experts
    (1500, 192, [170] + [80] * 7, TILED128, TILED128),
    (136, 128, [170] + [100] * 7, WIDE_KERNEL, TILED128),     # 130
    (136, 192, [170] + [100] * 7, WIDE_KERNEL, WIDE_KERNEL),
    (520, 192, [130] + [95] * 31, WIDE_KERNEL, WIDE_KERNEL),  # 116, 32 experts
    (520, 192, [130] + [95] * 30, TILED128, TILED128),
    (136, 128, [500] + [330] * 7, WIDE_KERNEL, TILED128),     # 389
    (136, 128, [500] + [400] * 7, WIDE_KERNEL, WIDE_KERNEL),  # 454
    (264, 192, [130] + [45] * 63, WIDE_KERNEL, WIDE_KERNEL),  # 60, many experts
    (264, 192, [130] + [56] * 63, TILED128, TILED128),        # 73
    (264, 192, [130] + [80] * 63, WIDE_KERNEL, WIDE_KERNEL),  # 99
    (264, 128, [140] + [80] * 63, WIDE_KERNEL, TILED128),     # 99
    (136, 128, [200] + [140] * 63, WIDE_KERNEL, WIDE_KERNEL), # 165
    (136, 192, [130] + [24] * 149, WIDE_KERNEL, TILED64),     # 35, as many experts as SMs
    (136, 192, [130] + [29] * 149, WIDE_KERNEL, WIDE_KERNEL), # 41
]


@pytest.mark.parametrize("O,rank,lengths,single,pair", REACHES)
def test_calls_reach_the_kernel_they_are_meant_for(lib, O, rank, lengths, single, pair):
    import trismoe_b200 as tm

    pa, pb = (_payload(tm, len(lengths), O, rank, 64, seed) for seed in (1, 2))
    h = torch.zeros((sum(lengths), rank), dtype=torch.float16, device="cuda")
    route = tm.qlinear_grouped._coerce_grouped_route(lengths, "cuda")
    for want, run in ((single, lambda: tm.run_grouped_structured_expert_forward(pa, h, None, route)),
                      (pair, lambda: tm.run_grouped_structured_expert_pair_forward(pa, pb, h, h, None, route, fuse_silu_mul=True))):
        run()
        names = [name for name, _ in kernels_of(run) if "grouped_" in name]
        assert len(names) == 1 and want in names[0], names


# Segments of many rows, unequal: one to six row tiles, more segments than a warp has lanes, columns that fit shared memory
# together (one or two chunks, the last one full or not) and columns that stream through it, an odd number of output tiles, as many
# segments as SMs; one to four row-scale slots a chunk, none to eight steps of salient columns, column scales.
WIDE = [
    (264, 256, 128, None, [300, 0, 5, 129, 700, 128]),
    (1040, 192, 128, None, [130 + 61 * (i % 7) for i in range(40)]),
    (136, 72, 128, None, [129, 513, 1]),
    (520, 328, 128, None, [257, 640, 384, 3]),
    (264, 1032, 128, None, [400, 129]),
    (136, 72, 128, None, [640, 513, 129]),
    (136, 192, 64, 0.1, [38 + i % 9 for i in range(150)]),
    (264, 256, 32, 0.0, [300, 131]),
    (264, 256, 32, 0.5, [131, 300]),
    (136, 328, 32, 0.97, [257, 140]),
    (264, 256, 64, 0.97, [300, 131]),
    (136, 328, 64, 0.5, [140, 257]),
    (136, 200, 96, 0.9, [300, 131]),
]


@pytest.mark.parametrize("O,rank,group,salient,lengths", WIDE)
def test_long_and_unequal_segments(lib, O, rank, group, salient, lengths):
    import trismoe_b200 as tm
    import trismoe_oracle as orc
    from trismoe_b200 import synth

    E, R = len(lengths), sum(lengths)
    more = {} if salient is None else {"p_salient": salient, "col_scale_one": False}
    pa, pb = _payload(tm, E, O, rank, group, O + rank, **more), _payload(tm, E, O, rank, group, O + rank + 1, **more)
    wa, wb = tm.dequantize_grouped_payload(pa), tm.dequantize_grouped_payload(pb)
    if more:  # groups and densities that no other test compares with the oracle
        p = synth.pack_projection(synth.raw_projection(np.random.default_rng(O + rank), E, O, rank, group_size=group, **more))
        assert np.array_equal(wa[E - 1].cpu().numpy(), orc.dequantize_expert(to_numpy_payload(p), E - 1))
    g = torch.Generator().manual_seed(R)
    ha, hb = ((0.5 * torch.randn((R, rank), generator=g)).half().cuda() for _ in range(2))
    route = tm.qlinear_grouped._coerce_grouped_route(lengths, "cuda")
    one = tm.run_grouped_structured_expert_forward(pa, ha, None, route)
    sa, sb = tm.run_grouped_structured_expert_pair_forward(pa, pb, ha, hb, None, route)
    ta, tb = tm.run_grouped_structured_expert_pair_forward(pa, pb, ha, ha, None, route)  # one set of rows
    mlp, _ = tm.run_grouped_structured_expert_pair_forward(pa, pb, ha, hb, None, route, fuse_silu_mul=True)
    row = 0
    for e, n in enumerate(lengths):
        if n == 0:
            continue
        rows = slice(row, row + n)
        row += n
        ra, ea, ba = _bound(wa[e], ha[rows])
        rb, eb, bb = _bound(wb[e], hb[rows])
        rc, _, bc = _bound(wb[e], ha[rows])
        for got, ref, bound in ((one, ra, ba), (sa, ra, ba), (sb, rb, bb), (ta, ra, ba), (tb, rc, bc)):
            _assert_within(got[rows], ref, bound)
        silu = ra * torch.sigmoid(ra)
        err = 1.1 * ea * rb.abs() + silu.abs() * eb + 1.1 * ea * eb + (silu * rb).abs() * (2.0 ** -11 + 2.0 ** -19) + 2.0 ** -25
        _assert_within(mlp[rows], silu * rb, err)
        for c in range(0, rank, n):  # one-hot rows: every weight exactly
            hot = torch.zeros_like(ha)
            hot[rows] = torch.nn.functional.one_hot((torch.arange(n, device="cuda") + c) % rank, rank).half()
            col = (torch.arange(n, device="cuda") + c) % rank
            assert torch.equal(tm.run_grouped_structured_expert_forward(pa, hot, None, route)[rows], wa[e][:, col].T)


@pytest.mark.parametrize("rank", [192, 328])
def test_long_segments_with_every_option(lib, rank):
    """Output scales and biases that differ by expert, gathered rows, a scale of the columns, outputs scattered or dropped, and rows
    further apart than they are long."""
    import ctypes as C

    import trismoe_b200 as tm
    from trismoe_b200 import synth

    lengths, O = [300, 129, 1, 200], 264
    E, R = len(lengths), sum(lengths)
    g = torch.Generator().manual_seed(rank)
    plain, payloads = [], []
    for seed in (5, 6):
        raw = synth.raw_projection(np.random.default_rng(seed), E, O, rank, group_size=64, col_scale_one=False)
        plain.append(tm.prepare_grouped_payload(synth.pack_projection(raw), "cuda"))
        p = synth.pack_projection(raw)
        p["output_scale"], p["has_output_scale"] = (1 + 0.2 * torch.randn((E, O), generator=g)).half(), True
        p["bias"], p["has_bias"] = (0.3 * torch.randn((E, O), generator=g)).half(), True
        payloads.append(tm.prepare_grouped_payload(p, "cuda"))
    expert = torch.repeat_interleave(torch.arange(E), torch.tensor(lengths)).cuda()
    route = dict(tm.qlinear_grouped._coerce_grouped_route(lengths, "cuda"))
    rows = (0.5 * torch.randn((57, rank), generator=g)).half().cuda()
    gather = torch.randint(0, 57, (R,), generator=g).to(torch.int32).cuda()
    scatter = torch.randperm(R, generator=g).to(torch.int32).cuda()
    scatter[::11] = -1
    col = (1 + 0.2 * torch.randn((rank,), generator=g)).half().cuda()
    kept = scatter >= 0
    h = rows[gather.long()]

    def check(x, p, outs, at):
        """One projection, both of a pair and SiLU * up of rows ``at`` against the dequantised matrices, output scale and bias."""
        refs = []
        for q in p:
            w = tm.dequantize_grouped_payload(q)
            ref, acc = torch.zeros((R, O), dtype=torch.float64, device="cuda"), torch.zeros((R, O), dtype=torch.float64, device="cuda")
            for e in range(E):
                ref[expert == e], acc[expert == e], _ = _bound(w[e], x[expert == e])
            if q["has_output_scale"]:
                sc, b = q["output_scale"].double()[expert], q["bias"].double()[expert]
                acc = acc * sc.abs() * (1 + 2.0 ** -22) + (ref * sc).abs() * 2.0 ** -22 + (ref * sc + b).abs() * 2.0 ** -22
                ref = ref * sc + b
            refs.append((ref[at], acc[at]))
        for got, (ref, acc) in zip(outs[:3], (refs[0], *refs)):
            _assert_within(got, ref, acc * (1 + 2.0 ** -10) + ref.abs() * 2.0 ** -11 + 2.0 ** -25)
        (ra, ea), (rb, eb) = refs
        silu = ra * torch.sigmoid(ra)
        err = 1.1 * ea * rb.abs() + silu.abs() * eb + 1.1 * ea * eb + (silu * rb).abs() * (2.0 ** -11 + 2.0 ** -19) + 2.0 ** -25
        _assert_within(outs[3], silu * rb, err)

    def run(p, x, r):
        one = tm.run_grouped_structured_expert_forward(p[0], x, None, r)
        return one, *tm.run_grouped_structured_expert_pair_forward(p[0], p[1], x, x, None, r), tm.run_grouped_structured_expert_pair_forward(p[0], p[1], x, x, None, r, fuse_silu_mul=True)[0]

    everything = torch.ones((R,), dtype=torch.bool, device="cuda")
    check(h, payloads, run(payloads, h, route), everything)
    check(h, payloads, run(payloads, rows, {**route, "_row_gather": gather}), everything)
    for p in (plain, payloads):
        check(h, p, [t[scatter[kept].long()] for t in run(p, h, {**route, "_out_row_scatter": scatter})], kept)
    scaled = (h.float() * col.float()).half()  # the product of two halves is rounded once
    check(scaled, payloads, run(payloads, h, {**route, "_hidden_col_scale": col}), everything)
    # rows 16 columns further apart, by tensor copies and (pair of two sets) without
    wide_rows = torch.full((R, rank + 16), float("nan"), dtype=torch.float16, device="cuda")
    wide_rows[:, :rank] = h
    want = run(payloads, h, route)
    keep, va, vb = [], tm.qlinear_grouped.proj_view(payloads[0]), tm.qlinear_grouped.proj_view(payloads[1])
    rv = tm.qlinear_grouped._route_view(route, R, keep)
    rv.hidden_row_stride = rank + 16
    got = [torch.empty_like(y) for y in want]
    stream = torch.cuda.current_stream().cuda_stream
    tm._native.check(lib.tris_grouped_forward(C.byref(va), C.byref(rv), wide_rows.data_ptr(), got[0].data_ptr(), stream))
    others = wide_rows.clone()
    tm._native.check(lib.tris_grouped_pair_forward(C.byref(va), C.byref(vb), C.byref(rv), wide_rows.data_ptr(), others.data_ptr(),
                                                   got[1].data_ptr(), got[2].data_ptr(), 0, stream))
    tm._native.check(lib.tris_grouped_pair_forward(C.byref(va), C.byref(vb), C.byref(rv), wide_rows.data_ptr(), wide_rows.data_ptr(),
                                                   got[3].data_ptr(), None, 1, stream))
    for y, w in zip(got, want):
        assert torch.equal(y, w)


@pytest.mark.parametrize("O,K,T", [(136, 520, 33), (137, 1100, 64), (1024, 2048, 65), (256, 4096, 130), (72, 8192, 300), (4096, 512, 257)])
def test_linear_columns_shared_among_ctas(lib, O, K, T):
    """An ordinary matrix of more than 32 rows: its columns in one to many parts, single and as a pair."""
    import trismoe_b200 as tm
    from trismoe_b200 import synth

    rng = np.random.default_rng(O + K)
    mods = []
    for _ in range(2):
        p = synth.pack_projection(synth.raw_projection(rng, 1, O, K, group_size=128))
        p["output_scale"] = torch.from_numpy((1 + 0.2 * rng.standard_normal((1, O))).astype(np.float16))
        p["has_output_scale"] = True
        mods.append(tm.Compact3Linear(p, device="cuda"))
    x = (0.5 * torch.randn((T, K), generator=torch.Generator().manual_seed(T))).half().cuda()
    refs = []
    for m in mods:
        w = tm.dequantize_grouped_payload(m.payload)[0]
        ref, err, _ = _bound(w, x)
        sc = m.payload["output_scale"].double().reshape(1, O)
        refs.append((ref * sc, err * sc.abs() * (1 + 2.0 ** -22) + (ref * sc).abs() * 2.0 ** -22))
    half = lambda r, e: e * (1 + 2.0 ** -10) + r.abs() * 2.0 ** -11 + 2.0 ** -25
    _assert_within(mods[0](x), refs[0][0], half(*refs[0]))
    a, b = tm.run_compact3_gate_up_forward(mods[0], mods[1], x, fuse_silu_mul=False)
    _assert_within(a, refs[0][0], half(*refs[0]))
    _assert_within(b, refs[1][0], half(*refs[1]))
    (ra, ea), (rb, eb) = refs
    silu = ra * torch.sigmoid(ra)
    err = 1.1 * ea * rb.abs() + silu.abs() * eb + 1.1 * ea * eb + (silu * rb).abs() * (2.0 ** -11 + 2.0 ** -19) + 2.0 ** -25
    _assert_within(tm.run_compact3_gate_up_forward(mods[0], mods[1], x), silu * rb, err)
    for c in range(0, K, T):  # one column of the matrix per row: exact but for the output scale's rounding
        col = (torch.arange(T, device="cuda") + c) % K
        hot = torch.nn.functional.one_hot(col, K).half()
        want = [(tm.dequantize_grouped_payload(m.payload)[0][:, col].float() * m.payload["output_scale"].float().view(O, 1)).half().t() for m in mods]
        a, b = tm.run_compact3_gate_up_forward(mods[0], mods[1], hot, fuse_silu_mul=False)
        assert torch.equal(mods[0](hot), want[0]) and torch.equal(a, want[0]) and torch.equal(b, want[1])


@pytest.mark.parametrize("O,K,T", [(40, 1024, 1), (33, 1040, 7), (136, 2300, 17), (72, 8192, 32), (1000, 1536, 24), (4096, 1100, 16), (96, 1288, 9)])
def test_linear_columns_shared_by_a_cluster(lib, O, K, T):
    """An ordinary matrix of up to 32 rows: its columns over two, four and eight CTAs, in equal and unequal parts; the bias once."""
    import trismoe_b200 as tm
    from trismoe_b200 import synth

    test_linear_columns_shared_among_ctas(lib, O, K, T)
    rng = np.random.default_rng(O)
    p = synth.pack_projection(synth.raw_projection(rng, 1, O, K, group_size=128))
    bias = torch.from_numpy(rng.standard_normal(O).astype(np.float16))
    lin = tm.Compact3Linear(p, bias=bias, device="cuda")
    x = (0.5 * torch.randn((T, K), generator=torch.Generator().manual_seed(T))).half().cuda()
    y = lin(x)
    ref, err, _ = _bound(tm.dequantize_grouped_payload(lin.payload)[0], x)
    ref = ref + bias.cuda().double()
    _assert_within(y, ref, err * (1 + 2.0 ** -10) + ref.abs() * (2.0 ** -11 + 2.0 ** -22) + 2.0 ** -25)
    assert all(torch.equal(lin(x), y) for _ in range(3))


@pytest.mark.parametrize("O,K,T,pair", [(1024, 2048, 256, False), (512, 2048, 512, True), (2048, 512, 300, False), (264, 1032, 129, True)])
def test_linear_parts_fill_the_gpu(lib, O, K, T, pair):
    """Rows in parts of 128, columns in as many parts as the SMs and two chunks a part allow."""
    import trismoe_b200 as tm
    from trismoe_b200 import synth

    rng = np.random.default_rng(1)
    mods = [tm.Compact3Linear(synth.pack_projection(synth.raw_projection(rng, 1, O, K, group_size=128)), device="cuda") for _ in range(2)]
    x = torch.zeros((T, K), dtype=torch.float16, device="cuda")
    run = (lambda: tm.run_compact3_gate_up_forward(*mods, x, fuse_silu_mul=False)) if pair else (lambda: mods[0](x))
    sms, tiles, chunks = torch.cuda.get_device_properties(0).multi_processor_count, -(-O // 128), -(-K // 128)
    units = tiles if pair else -(-tiles // 2)
    rows = min(4, sms // units, -(-T // 128))
    run()
    grids = [grid for name, grid in kernels_of(run) if "grouped_wide_kernel" in name]
    assert grids == [[units * rows * min(chunks // 2, sms // (units * rows)), 1, 1]]


@pytest.mark.parametrize("rows,cols,group,T", [
    (16, 32, 32, 1), (17, 40, 40, 8), (64, 64, 32, 9), (48, 96, 96, 17), (72, 128, 64, 33), (256, 264, 264, 65), (128, 2048, 128, 200),
])
def test_packed4_gemm_at_tile_edges(lib, rows, cols, group, T):
    import trismoe_b200 as tm
    import trismoe_oracle as orc
    from trismoe_b200 import synth

    m = synth.packed4_matrix(np.random.default_rng(rows + T), rows, cols, group_size=group, scale_std=0.02)
    lin = tm.Packed4Linear(m, "cuda")
    w = torch.from_numpy(orc.dequantize_packed4(*(m[k].numpy() for k in ("qweight", "qzeros", "scales", "g_idx")), rows, cols)).cuda()
    eye = torch.eye(cols, dtype=torch.float16, device="cuda")
    for c in range(0, cols, T):  # single products: the weights themselves, at this many rows
        assert torch.equal(lin(eye[c: c + T]), w.t()[c: c + T])
    g = torch.Generator().manual_seed(T)
    x = torch.randn((T, cols + 8), generator=g).half().cuda()
    for xi in (x[:, :cols].contiguous(), x[:, 3:3 + cols]):  # aligned rows, rows read element by element
        ref, _, bound = _bound(w, xi)
        _assert_within(lin(xi), ref, bound)


@pytest.mark.parametrize("T,H", [(1, 64), (3, 100), (70, 2048), (2, 4104)])
def test_shared_expert_add(lib, T, H):
    import trismoe_b200 as tm

    g = torch.Generator().manual_seed(H)
    x, routed, shared = (torch.randn((T, H), generator=g).half().cuda() for _ in range(3))
    w = (torch.randn((1, H), generator=g) * H ** -0.5).half().cuda()
    out = torch.empty_like(x)
    tm._native.check(lib.tris_shared_expert_add(x.data_ptr(), w.data_ptr(), routed.data_ptr(), shared.data_ptr(), T, H, out.data_ptr(),
                                                torch.cuda.current_stream().cuda_stream))
    z = (x.double() * w.double()).sum(1, keepdim=True)
    gate = torch.sigmoid(z)
    # the logit and the gate rounded to fp16 (|sigmoid'| <= 1/4), the product and the sum too
    err = shared.double().abs() * (z.abs() * 2.0 ** -13 + 2.0 ** -20 + gate * 2.0 ** -10) + (routed.double() + gate * shared.double()).abs() * 2.0 ** -10 + 2.0 ** -24
    _assert_within(out, routed.double() + gate * shared.double(), err)


@pytest.mark.parametrize("T", [1, 37, 300])
@pytest.mark.parametrize("pairs,scales", [("gate up down", ""), ("gate", "up"), ("up", "gate down"), ("down", "gate up down"), ("", "down")])
def test_null_space_and_input_scales_in_one_sequence(lib, T, pairs, scales):
    """The native layer sequence against the same block composed of the reference-named operators: both
    round gate, up, mlp and the routed rows to fp16, in the same places."""
    import trismoe_b200 as tm
    import trismoe_oracle as orc
    from trismoe_b200 import synth

    rng = np.random.default_rng(11)
    shape = synth.LayerShape(256, 192, 8, 2, rank=96, group_size=32)
    layer = synth.synth_layer(shape, seed=3)
    E, H, I = shape.num_experts, shape.hidden_size, shape.intermediate_size
    width = {"gate": H, "up": H, "down": I}
    vec = {n: torch.from_numpy((1 + 0.2 * rng.standard_normal(width[n])).astype(np.float16)) for n in scales.split()}
    blk = tm.TrisSparseMoeBlock(H, I, E, shape.top_k, shape.norm_topk_prob)
    blk.load_grouped_payloads(layer["gate"], layer["up"], layer["down"], layer["shared_gate"], layer["shared_up"], layer["shared_down"],
                              layer["router_weight"], device="cuda", input_scales=vec)

    def pair(n):
        out = H if n == "down" else I
        ex = [None if r == 0 else {"c2": synth.packed4_matrix(rng, r, width[n], 64, scale_std=0.02),
                                   "c1": synth.packed4_matrix(rng, out, r, 64, scale_std=0.02)} for r in (16, 0, 24, 16, 8, 40, 0, 16)]
        return tm.build_grouped_ns_compensation_payload(ex, "cuda", torch.float16, width[n], out)

    blk.load_ns_compensation_payloads(*(pair(n) if n in pairs.split() else None for n in ("gate", "up", "down")))
    x = synth.synth_activations(T, H, seed=T).cuda().view(1, T, -1)
    logits = synth.synth_router_logits(T, E, seed=T).cuda()
    want, l_ops = blk.forward_grouped_ops(x, router_logits=logits)
    got, l_got = blk(x, router_logits=logits)
    assert l_got is logits and l_ops is logits
    max_abs, mean_rel = orc.error_metrics(got.float().cpu().numpy(), want.float().cpu().numpy())
    # routing weights stay fp32 in the sequence (fp16 in the composed operators: 2^-11), gate/up without a
    # pair stay fp32 before SiLU (fp16 there: 2^-11 each): four roundings of 2^-11 that one side has alone
    scale = want.float().abs().max().item()
    assert want.abs().max() > 1e-3 and max_abs <= 8 * 2.0 ** -11 * scale and mean_rel <= 4 * 2.0 ** -11, (max_abs, mean_rel, scale)
    _, own = blk(x)
    assert own.dtype == torch.float16 and own.shape == (T, E)


@pytest.mark.parametrize("T", [3, 40])
@pytest.mark.parametrize("counts", [[192, 64, 37, 0, 130, 1, 95, 191]])
def test_null_space_pair_of_up_with_fewer_outputs_than_gate(lib, T, counts):
    """Outputs that up's pair does not reach are up's own, and SiLU(gate) * up is theirs as well: the bits of a pair whose scales are zero there."""
    import trismoe_b200 as tm
    from trismoe_b200 import synth

    shape = synth.LayerShape(256, 192, 8, 2, rank=96, group_size=32)
    layer = synth.synth_layer(shape, seed=3)
    E, H, I = shape.num_experts, shape.hidden_size, shape.intermediate_size
    x, logits = synth.synth_activations(T, H, seed=T).cuda().view(1, T, -1), synth.synth_router_logits(T, E, seed=T).cuda()
    outs = []
    for by_scales in (True, False):
        rng = np.random.default_rng(19)
        blk = tm.TrisSparseMoeBlock(H, I, E, shape.top_k, shape.norm_topk_prob)
        blk.load_grouped_payloads(*({k: v.clone() if isinstance(v, torch.Tensor) else v for k, v in layer[n].items()} for n in ("gate", "up", "down")),
                                  layer["shared_gate"], layer["shared_up"], layer["shared_down"], layer["router_weight"], device="cuda")
        pairs = []
        for which in range(2):
            ex = [{"c2": synth.packed4_matrix(rng, 32, H, 64, scale_std=0.02), "c1": synth.packed4_matrix(rng, I, 32, 64, scale_std=0.02)} for _ in range(E)]
            for e in range(E):
                if which and by_scales:
                    ex[e]["c1"]["scales"][..., counts[e]:] = 0
            pairs.append(tm.build_grouped_ns_compensation_payload(ex, "cuda", torch.float16, H, I))
        blk.load_ns_compensation_payloads(pairs[0], pairs[1], None)
        blk._layer_extras(x.device)  # prepares the views
        counts_dev = torch.tensor(counts, dtype=torch.int32, device="cuda")
        if not by_scales:
            pairs[1]["_tris_c1_view"].n_count = counts_dev.data_ptr()
        outs.append(blk(x, router_logits=logits)[0])
        torch.cuda.synchronize()
    assert torch.equal(*outs) and outs[0].float().abs().max() > 1e-3


@pytest.mark.parametrize("T", [1, 8, 32, 70, 300])
@pytest.mark.parametrize("pairs,given", [("gate up down", True), ("gate up down", False), ("down", True), ("up", False)])
def test_null_space_layers_back_to_back(lib, T, pairs, given):
    """Products that start beside the launch ahead of them read rows, route and intermediate results before their wait: in calls with other
    rows each, nothing between them, eager and replayed, every result is that of the same call by itself."""
    import trismoe_b200 as tm
    from trismoe_b200 import synth

    rng = np.random.default_rng(17)
    E, H, I = 16, 512, 256
    layer = synth.synth_layer(synth.LayerShape(H, I, E, 4, rank=96, group_size=32), seed=5)
    blk = tm.TrisSparseMoeBlock(H, I, E, 4, True)
    blk.load_grouped_payloads(layer["gate"], layer["up"], layer["down"], layer["shared_gate"], layer["shared_up"], layer["shared_down"],
                              layer["router_weight"], device="cuda")

    def pair(n):
        width, out = (I, H) if n == "down" else (H, I)
        ex = [{"c2": synth.packed4_matrix(rng, r, width, 64, scale_std=0.02), "c1": synth.packed4_matrix(rng, out, r, 64, scale_std=0.02)}
              for r in rng.choice([16, 32, 64], E)]
        return tm.build_grouped_ns_compensation_payload(ex, "cuda", torch.float16, width, out)

    blk.load_ns_compensation_payloads(*(pair(n) if n in pairs.split() else None for n in ("gate", "up", "down")))
    xs = [synth.synth_activations(T, H, seed=10 * T + i).cuda().view(1, T, H) for i in range(4)]
    logits = [synth.synth_router_logits(T, E, seed=20 * T + i).cuda() if given else None for i in range(4)]
    want = []
    for x, l in zip(xs, logits):
        torch.cuda.synchronize()
        want.append(blk(x, router_logits=l)[0].clone())
        torch.cuda.synchronize()
    assert not any(torch.equal(want[0], w) for w in want[1:])
    got = [blk(x, router_logits=l)[0] for _ in range(8) for x, l in zip(xs, logits)]
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i % 4]) for i, y in enumerate(got))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = [blk(x, router_logits=l)[0] for x, l in zip(xs, logits)]
    for _ in range(5):
        for y in captured:
            y.fill_(7.0)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for y, w in zip(captured, want))


@pytest.mark.parametrize("T", [3, 37, 100])
@pytest.mark.parametrize("packed", ["gate up down", "gate up", "down"])
@pytest.mark.parametrize("pairs,scales", [("gate up down", "gate up down"), ("", "gate"), ("up", "up"), ("down", "gate up"), ("gate", "down"), ("gate up", "")])
def test_null_space_and_input_scales_with_4_bit_backbones(lib, T, packed, pairs, scales):
    """The form checkpoints arrive in: backbones kept as nibbles (up to 64 rows; routed rows cross that earlier) or
    expanded for the call, with scales and pairs on any of the projections."""
    import trismoe_b200 as tm
    import trismoe_oracle as orc
    from trismoe_b200 import synth

    rng = np.random.default_rng(13)
    shape = synth.LayerShape(256, 192, 8, 2, rank=96, group_size=32)
    layer = synth.synth_layer(shape, seed=4)
    E, H, I = shape.num_experts, shape.hidden_size, shape.intermediate_size
    width = {"gate": H, "up": H, "down": I}
    backbone = {n: synth.packed4_matrix(rng, 96, width[n], 64, scale_std=0.02) if n in packed.split() else layer["shared_" + n] for n in width}
    vec = {n: torch.from_numpy((1 + 0.2 * rng.standard_normal(width[n])).astype(np.float16)) for n in scales.split()}
    blk = tm.TrisSparseMoeBlock(H, I, E, shape.top_k, shape.norm_topk_prob)
    blk.load_grouped_payloads(layer["gate"], layer["up"], layer["down"], backbone["gate"], backbone["up"], backbone["down"],
                              layer["router_weight"], device="cuda", input_scales=vec)
    assert set(blk.packed_backbones) == set(packed.split())

    def pair(n):
        out = H if n == "down" else I
        ex = [None if r == 0 else {"c2": synth.packed4_matrix(rng, r, width[n], 64, scale_std=0.02),
                                   "c1": synth.packed4_matrix(rng, out, r, 64, scale_std=0.02)} for r in (16, 0, 24, 16, 8, 40, 0, 16)]
        return tm.build_grouped_ns_compensation_payload(ex, "cuda", torch.float16, width[n], out)

    blk.load_ns_compensation_payloads(*(pair(n) if n in pairs.split() else None for n in ("gate", "up", "down")))
    x = synth.synth_activations(T, H, seed=T).cuda().view(1, T, -1)
    logits = synth.synth_router_logits(T, E, seed=T).cuda()
    want, _ = blk.forward_grouped_ops(x, router_logits=logits)
    for _ in range(2):
        got, _ = blk(x, router_logits=logits)
        max_abs, mean_rel = orc.error_metrics(got.float().cpu().numpy(), want.float().cpu().numpy())
        # the roundings that one side has alone, as in the test above
        scale = want.float().abs().max().item()
        assert want.abs().max() > 1e-3 and max_abs <= 8 * 2.0 ** -11 * scale and mean_rel <= 4 * 2.0 ** -11, (max_abs, mean_rel, scale)
    blk.raise_on_kernel_status()


@pytest.mark.parametrize("E,k", [(8, 2), (40, 8), (72, 3), (200, 8)])
@pytest.mark.parametrize("T", [1, 31, 32, 33, 65, 128, 225, 255, 256, 257, 2100])
def test_router_and_route_of_the_layer(lib, E, k, T):
    """One CTA up to 32 tokens, a cluster of up to eight to 256 (the last group ragged or full), two launches above, runs of several 32-token
    groups per CTA above 2048; expert counts on both sides of each lane count.  An identity-like layer would hide a wrong order, so whole outputs are compared."""
    import trismoe_b200 as tm
    import trismoe_oracle as orc
    from trismoe_b200 import synth

    shape = synth.LayerShape(64, 64, E, k, rank=32, group_size=32)
    layer = synth.synth_layer(shape, seed=E)
    blk = tm.TrisSparseMoeBlock(64, 64, E, k, shape.norm_topk_prob)
    blk.load_grouped_payloads(layer["gate"], layer["up"], layer["down"], *(10 * layer["shared_" + n] for n in ("gate", "up", "down")),
                              layer["router_weight"], device="cuda")
    x, logits = synth.synth_activations(T, 64, seed=T).cuda().view(1, T, 64), synth.synth_router_logits(T, E, seed=T).cuda()
    want, _ = blk.forward_grouped_ops(x, router_logits=logits)
    got, _ = blk(x, router_logits=logits)
    scale = want.float().abs().max().item()
    max_abs, mean_rel = orc.error_metrics(got.float().cpu().numpy(), want.float().cpu().numpy())
    # what the composed operators round to fp16 and the sequence does not: gate, up, SiLU, routing weight, weighted row
    assert scale > 1e-3 and max_abs <= 10 * 2.0 ** -11 * scale and mean_rel <= 5 * 2.0 ** -11, (max_abs, mean_rel, scale)


# 64- and 128-row tiles of the backbone GEMM: ragged rows, outputs and columns, one to many row tiles.  128: more tiles than SMs, two
# to sixteen chunks of columns in a ring of three (as many as SMs exactly: 64); long rows whose columns are split into fours and eights.  73 clusters
# of four do not run at once, nor are eighths of 8192 columns long enough: 64.
@pytest.mark.parametrize("n,k,m,tile", [
    (33, 64, 64, None), (127, 192, 72, 64), (129, 1032, 256, None), (300, 2048, 136, 64), (1025, 512, 264, 64), (2048, 1024, 128, 64),
    (9601, 128, 256, 128), (9601, 256, 250, 128), (9601, 1024, 256, 128), (9472, 512, 256, 64), (2480, 8192, 256, 128), (1500, 10240, 200, 128), (1500, 8192, 256, 64), (9304, 8192, 128, 64),
])
def test_backbone_gemm_at_tile_edges(lib, n, k, m, tile):
    import trismoe_b200 as tm

    g = torch.Generator().manual_seed(n + m)
    x = torch.randn((n, k), generator=g).half().cuda()
    w = (0.05 * torch.randn((m, k), generator=g)).half().cuda()
    ref, _, bound = _bound(w, x)
    _assert_within(tm.compute_shared_hidden(x, w), ref, bound)
    if tile is not None:
        (name, _), = kernels_of(lambda: tm.compute_shared_hidden(x, w))
        assert "umma_gemm_tma_kernel<%d>" % tile in name
    for c in range(0, k, n):
        col = (torch.arange(n, device="cuda") + c) % k
        assert torch.equal(tm.compute_shared_hidden(torch.nn.functional.one_hot(col, k).half(), w), w.t()[col])


# Tiles of 128 rows x 256 outputs, taken by launches that overlap their predecessor: ragged rows, one to several tiles of outputs (the last one
# narrow), two to many chunks of columns in a ring of four, columns in halves and quarters, two turns of tiles.
@pytest.mark.parametrize("n,k,ms", [(5100, 128, [256]), (6145, 192, [250]), (5200, 1024, [300]), (17000, 64, [320]), (10400, 320, [128]), (2048, 2048, [256, 256, 64]),
                                    (1793, 4096, [256, 256, 8]), (3000, 8192, [256]), (2100, 2112, [264, 264, 250])])
def test_backbone_gemm_in_big_tiles(lib, n, k, ms):
    import trismoe_b200 as tm

    g = torch.Generator().manual_seed(n + k)
    x = torch.randn((n, k), generator=g).half().cuda()
    ws = [(0.05 * torch.randn((m, k), generator=g)).half().cuda() for m in ms]

    def run(x):
        if len(ws) == 1:
            return [tm.compute_shared_hidden(x, ws[0])]
        # two matrices and a router of one launch
        outs = [torch.empty((n, m), dtype=torch.float16 if i < 2 else torch.float32, device="cuda") for i, m in enumerate(ms)]
        tm._native.check(lib.tris_input_projections(x.data_ptr(), n, k, ws[0].data_ptr(), ws[1].data_ptr(), ms[0], ws[2].data_ptr(), ms[2], outs[0].data_ptr(),
                                                    outs[1].data_ptr(), 0, outs[2].data_ptr(), torch.cuda.current_stream().cuda_stream))
        return outs

    previous = lib.tris_set_programmatic_launch(1)
    try:
        outs = run(x)
        names = [name for name, _ in kernels_of(lambda: run(x))]
        hots = []
        for c in range(0, k, n):
            col = (torch.arange(n, device="cuda") + c) % k
            hots.append((col, run(torch.nn.functional.one_hot(col, k).half())))
        if ms[0] % 32 == 0 and len(ws) == 1:
            plain, permuted = outs[0], tm.compute_shared_hidden(x, ws[0], layout=2)
    finally:
        lib.tris_set_programmatic_launch(previous)
    assert any("umma_gemm_big_kernel" in name for name in names), names
    for got, w in zip(outs, ws):
        ref, acc, bound = _bound(w, x)
        _assert_within(got, ref, bound if got.dtype == torch.float16 else acc + 2.0 ** -25)
    for col, outs in hots:
        for got, w in zip(outs, ws):
            assert torch.equal(got, w.t()[col].to(got.dtype))
    if ms[0] % 32 == 0 and len(ws) == 1:
        at = torch.arange(ms[0])
        place = (at & ~31) | ((at & 15) << 1) | ((at >> 4) & 1)
        assert torch.equal(permuted[:, place.cuda()], plain)


@pytest.mark.parametrize("n,k,m", [(2480, 8192, 256), (1880, 8192, 250), (4000, 8192, 128), (1200, 8192, 128)])
def test_backbone_gemm_of_gathered_long_rows(lib, n, k, m):
    import trismoe_b200 as tm

    g = torch.Generator().manual_seed(n + m)
    rows = torch.randn((300, k), generator=g).half().cuda()
    w = (0.05 * torch.randn((m, k), generator=g)).half().cuda()
    gather = torch.randint(0, 300, (n,), generator=g).to(torch.int32).cuda()
    out = torch.empty((n, m), dtype=torch.float16, device="cuda")
    tm._native.check(lib.tris_shared_hidden_forward(rows.data_ptr(), gather.data_ptr(), n, None, k, w.data_ptr(), m, out.data_ptr(), 0,
                                                    torch.cuda.current_stream().cuda_stream))
    ref, _, bound = _bound(w, rows)
    _assert_within(out, ref[gather.long()], bound[gather.long()])


@pytest.mark.parametrize("T", [1, 16, 70])
def test_batch_whose_logits_are_not_numbers(lib, T):
    """No segment has rows: every launch of the sequence still waits for the one before, the outputs are not numbers
    either and the next batch is computed as ever."""
    import trismoe_b200 as tm
    from trismoe_b200 import synth

    shape = synth.LayerShape(256, 192, 8, 2, rank=96, group_size=32)
    layer = synth.synth_layer(shape, seed=5)
    blk = tm.TrisSparseMoeBlock(256, 192, 8, 2, True)
    blk.load_grouped_payloads(layer["gate"], layer["up"], layer["down"], layer["shared_gate"], layer["shared_up"], layer["shared_down"],
                              layer["router_weight"], device="cuda")
    x, logits = synth.synth_activations(T, 256, seed=T).cuda().view(1, T, 256), synth.synth_router_logits(T, 8, seed=T).cuda()
    want = blk(x, logits)[0].clone()
    for _ in range(3):
        assert blk(x, torch.full_like(logits, float("nan")))[0].isnan().all()
        assert torch.equal(blk(x, logits)[0], want)


@pytest.mark.parametrize("rank", [32, 96, 256, 320])
@pytest.mark.parametrize("lengths", [[1, 5, 0, 16], [40, 3, 64, 33], [130, 70]])
@pytest.mark.parametrize("offset", [0, 4])
def test_permuted_rows_give_the_same_bits(lib, rank, lengths, offset):
    """Rows in the two permuted column orders, at 16-byte boundaries and off them, against the same rows row-major."""
    import trismoe_b200 as tm

    E, R, O = len(lengths), sum(lengths), 104
    pa, pb = _payload(tm, E, O, rank, 32, rank), _payload(tm, E, O, rank, 32, rank + 1)
    rows = (0.5 * torch.randn((R, rank), generator=torch.Generator().manual_seed(R))).half().cuda()
    eye = torch.eye(rank, dtype=torch.float16, device="cuda")
    route = dict(tm.qlinear_grouped._coerce_grouped_route(lengths, "cuda"))
    run = lambda h, r: (tm.run_grouped_structured_expert_forward(pa, h, None, r),
                        *tm.run_grouped_structured_expert_pair_forward(pa, pb, h, h, None, r),
                        tm.run_grouped_structured_expert_pair_forward(pa, pb, h, h, None, r, fuse_silu_mul=True)[0])
    want = run(rows, route)
    for layout in (tm.HIDDEN_PAIR_INTERLEAVED, tm.HIDDEN_LANE_ORDER):
        buf = torch.empty((R * rank + 8,), dtype=torch.float16, device="cuda")
        h = buf[offset: offset + R * rank].view(R, rank)
        h.copy_(tm.compute_shared_hidden(rows, eye, layout=layout))  # single products: the rows themselves, permuted
        for a, b in zip(run(h, {**route, "_hidden_layout": layout}), want):
            assert torch.equal(a, b)


def test_pair_of_ordinary_linears_of_which_one_has_no_records(lib):
    import trismoe_b200 as tm
    from trismoe_b200 import synth

    rng = np.random.default_rng(7)
    mods = []
    for records in (True, False):
        p = synth.pack_projection(synth.raw_projection(rng, 1, 96, 512, group_size=128))
        mods.append(tm.Compact3Linear(tm.prepare_grouped_payload(p, "cuda", tile_records=records)))
    x = (0.5 * torch.randn((5, 512), generator=torch.Generator().manual_seed(5))).half().cuda()
    for pair in (mods, mods[::-1]):
        for y, m in zip(tm.run_compact3_gate_up_forward(*pair, x, fuse_silu_mul=False), pair):
            ref, _, bound = _bound(tm.dequantize_grouped_payload(m.payload)[0], x)
            _assert_within(y, ref, bound)
