"""GPU: memory that a call has handed to the device stays untouched until the device is through with it -- also
when the caller drops or changes it right after the (asynchronous) call."""
import pytest
import torch

from conftest import assert_close
from oracle import acsr_oracle as ao
from oracle import attention_oracle as at

pytestmark = pytest.mark.gpu

SLEEP = 400_000_000      # SM clocks, some 0.2 s: what is queued behind it has not begun when the host goes on


def test_forward_host_operands_may_be_dropped():
    """Page-locked operands that the caller drops after forward_host returns are not handed out again before they
    have been copied, and a dropped result is not written into somebody else's block."""
    import acsr_helpers as ah
    import r_attention
    B, H, L, d = 1, 4, 1024, 64
    attn = r_attention.RegularAttention(B, L, H, d, ah.create_causal_windowed_mask(L, 100), 16, 16, 0, torch.bfloat16)
    torch.manual_seed(3)
    q, k, v = (torch.randn(B, H, L, d).to(torch.bfloat16) for _ in range(3))
    out = torch.empty(B, H, L, d, dtype=torch.bfloat16).pin_memory()
    attn.forward_host(q.pin_memory(), k.pin_memory(), v.pin_memory(), out)
    torch.cuda.synchronize()
    expected, out = out.clone(), torch.zeros_like(out).pin_memory()
    torch.cuda._sleep(SLEEP)
    attn.forward_host(q.pin_memory(), k.pin_memory(), v.pin_memory(), out)
    others = [torch.full((B, H, L, d), float("nan"), dtype=torch.bfloat16).pin_memory() for _ in range(6)]
    torch.cuda.synchronize()
    assert torch.equal(out, expected)
    del others
    torch.cuda._sleep(SLEEP)
    attn.forward_host(q.pin_memory(), k.pin_memory(), v.pin_memory(), torch.zeros_like(out).pin_memory())
    others = [torch.full((B, H, L, d), 7.0, dtype=torch.bfloat16).pin_memory() for _ in range(6)]
    torch.cuda.synchronize()
    assert all((t == 7).all() for t in others)


def test_captured_calls_follow_their_metadata():
    """A replayed graph works with the metadata that the tensors hold at the replay, like any other operand."""
    import acsr_helpers as ah
    import r_attention
    import splat_native as n
    L, H, d, dtype = 640, 2, 64, torch.bfloat16
    attn = r_attention.RegularAttention(1, L, H, d, ah.create_causal_windowed_mask(L, 200), 16, 16, 0, dtype, scale=0.125)
    acsr = ah.create_acsr(ah.create_causal_windowed_mask(L, 200), 16, 0)
    torch.manual_seed(4)
    q, k, v = (torch.randn(1, H, L, d).to(dtype) for _ in range(3))
    qd, vd, kt = q.cuda(), v.cuda(), k.cuda().transpose(2, 3)
    s = torch.empty(1, H, L, acsr[5], dtype=dtype, device="cuda")
    p = torch.rand(1, H, L, acsr[5]).to(dtype)
    pd, o = p.cuda(), torch.empty_like(qd)

    def calls():
        fused = attn([qd, kt, vd])
        n.sddmm(qd, kt, s, acsr[2], acsr[3], acsr[4], acsr[5])
        n.spmm(pd, vd, o, acsr[2], acsr[3], acsr[4], acsr[5])
        return fused

    calls()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fused = calls()
    narrow = ah.create_acsr(ah.create_causal_windowed_mask(L, 70), 16, 0)
    for i, name in ((2, "sTod_linear_transformations"), (3, "sTod_translations"), (4, "nnzs")):
        getattr(attn, name).copy_(narrow[i])
        acsr[i].copy_(narrow[i])
    graph.replay()
    torch.cuda.synchronize()
    meta = ao.metadata_from_pattern(ao.PATTERN_CAUSAL_WINDOWED, L, 70, 0, 16)
    assert_close(fused, at.attention_acsr(q, k.transpose(2, 3), v, meta, meta["trailing_dim"], 0.125), dtype, "fused")
    assert_close(s, at.sddmm_acsr(q, k.transpose(2, 3), meta, acsr[5]), dtype, "sddmm")
    assert_close(o, at.spmm_acsr(p, v, meta), dtype, "spmm")


@pytest.mark.parametrize("call", ["module", "sddmm"])
def test_band_table_of_a_call_on_another_stream(call):
    """Metadata dropped while a call on a side stream waits: the caller records the tensors it knows of, the table
    behind them has to last as long."""
    import acsr_helpers as ah
    import r_attention
    import splat_native as n
    L, H, d, dtype = 640, 2, 64, torch.bfloat16
    attn = r_attention.RegularAttention(1, L, H, d, ah.create_causal_windowed_mask(L, 200), 16, 16, 0, dtype, scale=0.125)
    T, side = attn.acsr_trailing_dim, torch.cuda.Stream()
    q, k, v = (torch.randn(1, H, L, d, device="cuda").to(dtype) for _ in range(3))
    s = torch.empty(1, H, L, T, dtype=dtype, device="cuda")

    def run():
        if call == "module":
            return attn([q, k.transpose(2, 3), v])
        n.sddmm(q, k.transpose(2, 3), s, attn.sTod_linear_transformations, attn.sTod_translations, attn.nnzs, T)
        return s

    expected = run().clone()
    torch.cuda.synchronize()
    size = attn.nnzs._splat_plan[4].numel()
    with torch.cuda.stream(side):
        torch.cuda._sleep(SLEEP)
        out = run()
    for t in (attn.sTod_linear_transformations, attn.sTod_translations, attn.nnzs):
        t.record_stream(side)
    del attn, t
    others = [torch.zeros(size, dtype=torch.int32, device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    assert torch.equal(out, expected) and all((t == 0).all() for t in others)
