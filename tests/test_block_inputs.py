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
