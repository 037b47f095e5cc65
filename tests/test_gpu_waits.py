"""GPU: the bounded waits of the tensor-core kernels and what a set status word does -- to a launch, and to a persistent
kernel that is already running.  Nothing here hangs or faults: the one wait that runs out has a short limit."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _selftest(word, limit_cycles):
    import splat_native as n
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    assert n._lib.splat_selftest_bounded_wait(word.data_ptr(), limit_cycles, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    return time.perf_counter() - t0


def test_waits_give_up_after_their_limit():
    """Three waits of 1e8 cycles (some 50 ms) each: within a factor of four, and never without waiting."""
    word = torch.zeros(1, dtype=torch.int32, device="cuda")
    seconds = _selftest(word, 100_000_000)
    assert word.item() == 99
    assert 0.15 / 4 < seconds < 0.15 * 4


def test_a_status_word_that_is_set_stays():
    word = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    _selftest(word, 1000)
    assert word.item() == 7


def _calls():
    """(name, launch(out), out) of every default tensor-core kernel."""
    import acsr_helpers as ah
    import splat_native as n
    H, L = 74, 2048                                      # 1184 tiles: the persistent kernel at d = 128
    acsr = ah.create_acsr(ah.create_causal_windowed_mask(L, 63), 16, 0)
    meta, T = (acsr[2], acsr[3], acsr[4]), acsr[5]
    for d in (64, 128):
        x = torch.randn(1, H, L, d, device="cuda").to(torch.bfloat16)
        p = torch.rand(1, H, L, T, device="cuda").to(torch.bfloat16)
        yield f"fused d={d}", lambda o, x=x: n.attention_fused(x, x.transpose(2, 3), x, o, *meta, 0.125, n.PATH_BAND), torch.empty_like(x)
        yield f"sddmm d={d}", lambda o, x=x: n.sddmm(x, x.transpose(2, 3), o, *meta, T), torch.empty_like(p)
        yield f"spmm d={d}", lambda o, x=x, p=p: n.spmm(p, x, o, *meta, T), torch.empty_like(x)


def test_launches_do_nothing_while_the_status_word_is_set():
    import splat_native as n
    for name, launch, out in _calls():
        out.fill_(3.0)
        launch(out)
        n.check_status_word(0)
        assert not (out == 3.0).all(), name
        n.status_word(torch.device("cuda", 0)).fill_(7)
        out.fill_(3.0)
        launch(out)
        torch.cuda.synchronize()
        assert (out == 3.0).all(), name
        with pytest.raises(RuntimeError):
            n.check_status_word(0)                       # reports and clears
        launch(out)
        n.check_status_word(0)
        assert torch.isfinite(out.float()).all(), name


def test_running_kernel_stops_when_the_status_word_is_set():
    """A CTA that has not begun when another gives up does no work; a persistent CTA that is running takes no more tiles."""
    import acsr_helpers as ah
    import splat_native as n
    H, L, d = 256, 32768, 128                            # some 5 ms
    acsr = ah.create_acsr(ah.create_causal_windowed_mask(L, 1023), 16, 0)
    q = torch.randn(1, 1, L, d, device="cuda").to(torch.bfloat16).expand(1, H, L, d).contiguous()
    out = torch.empty_like(q)
    word, five, side = n.status_word(torch.device("cuda", 0)), torch.full((1,), 5, dtype=torch.int32).pin_memory(), torch.cuda.Stream()

    def launch():
        n.attention_fused(q, q.transpose(2, 3), q, out, acsr[2], acsr[3], acsr[4], d ** -0.5, n.PATH_BAND)

    launch()
    n.check_status_word(0)
    seen = []
    for _ in range(5):
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        launch()
        done = torch.cuda.Event()
        done.record()
        until = time.perf_counter() + 1e-3
        while time.perf_counter() < until:
            pass
        with torch.cuda.stream(side):                    # (by a copy engine: the SMs are full)
            word.copy_(five, non_blocking=True)
        side.synchronize()
        in_time = not done.query()
        torch.cuda.synchronize()
        first, last = torch.isfinite(out[0, 0].float()).all().item(), torch.isfinite(out[0, -1].float()).all().item()
        with pytest.raises(RuntimeError):
            n.check_status_word(0)
        if in_time:
            seen.append((first, last))
            if (first, last) == (True, False):
                break
    if not seen:
        pytest.skip("the word was never set while the kernel ran")
    assert (True, False) in seen
