"""GPU: memory that a call has handed to the device stays untouched until the device is through with it -- also
when the caller drops or changes it right after the (asynchronous) call."""
import pytest
import torch

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
