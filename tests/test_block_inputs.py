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
