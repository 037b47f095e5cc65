"""GPU: calls that something stands in the way of -- no memory for a copy, nothing set up yet, unusual operands -- give
what the ordinary calls give."""
import subprocess
import sys
import textwrap

import pytest
import torch

from conftest import ROOT, SPLAT_DIR

pytestmark = pytest.mark.gpu


def run_python(code, *flags):
    """In a process of its own: nothing warmed up, no state of other tests."""
    head = f"import sys; sys.path[:0] = [{ROOT!r}, {SPLAT_DIR!r}, {ROOT + '/tests'!r}]\nimport torch\n"
    return subprocess.run([sys.executable, *flags, "-c", head + textwrap.dedent(code)], capture_output=True, text=True, timeout=300)


@pytest.mark.parametrize("call", ["module", "sddmm"])
def test_out_of_memory_for_the_copy_of_kt(call):
    """No room for the row-major copy of a contiguous K^T: the kernels that need none run."""
    r = run_python(f"""
        import acsr_helpers as ah, r_attention, splat_native as n
        B, H, L, d = 1, 64, 4096, 64
        attn = r_attention.RegularAttention(B, L, H, d, ah.create_strided_mask(L, 64), 16, 16, 0, torch.bfloat16, scale=0.125)
        T = attn.acsr_trailing_dim
        q, v = (torch.randn(B, H, L, d, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        kt = torch.randn(B, H, d, L, dtype=torch.bfloat16, device="cuda")
        s = torch.empty(B, H, L, T, dtype=torch.bfloat16, device="cuda")
        meta = attn.sTod_linear_transformations, attn.sTod_translations, attn.nnzs
        def call():
            if {call!r} == "module":
                return attn([q, kt, v]).clone()
            n.sddmm(q, kt, s, *meta, T)
            return s.clone()
        expected = call()
        call()
        hold = torch.empty_like(expected)
        torch.cuda.synchronize(); torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (8 << 20)) / total)
        if {call!r} == "module":
            hold.copy_(attn([q, kt, v]))
        else:
            n.sddmm(q, kt, s, *meta, T)
            hold.copy_(s)
        torch.cuda.synchronize()
        torch.cuda.set_per_process_memory_fraction(1.0)
        assert (hold.float() - expected.float()).abs().max() < 5e-2 * max(1.0, expected.float().abs().max().item())
        print("fine")
        """)
    assert r.returncode == 0 and "fine" in r.stdout, (r.returncode, r.stderr[-2000:])


def test_operands_without_data():
    """Fake and sparse tensors: an exception."""
    import acsr_helpers as ah
    import r_attention
    from torch._subclasses.fake_tensor import FakeTensorMode
    attn = r_attention.RegularAttention(1, 64, 1, 64, ah.create_causal_windowed_mask(64, 8), 16, 16, 0, torch.float16)
    x = torch.randn(1, 1, 64, 64, dtype=torch.float16, device="cuda")
    attn([x, x.transpose(2, 3), x])
    with FakeTensorMode(allow_non_fake_inputs=True) as mode:
        f = mode.from_tensor(x)
        with pytest.raises(Exception):
            attn([f, f.transpose(2, 3), f])
    with pytest.raises(Exception):
        attn([x.to_sparse(), x.transpose(2, 3), x])


def test_first_fp32_launchers_under_capture():
    """The fp32 launchers and the softmax of any type need nothing from the device but their operands: a process may
    capture its very first calls."""
    r = run_python("""
        import acsr_helpers as ah, splat_native as n
        from conftest import assert_close
        from oracle import acsr_oracle as ao, attention_oracle as at
        L, H, d = 300, 2, 64
        acsr = ah.create_acsr(ah.create_causal_windowed_mask(L, 40), 16, 0)
        torch.manual_seed(1)
        q, k, v = (torch.randn(1, H, L, d) for _ in range(3))
        qd, kt, vd = q.cuda(), k.cuda().transpose(2, 3), v.cuda()
        s = torch.empty(1, H, L, acsr[5], device="cuda")
        p, o = torch.empty_like(s), torch.empty_like(qd)
        x16 = torch.randn(1, H, L, acsr[5], dtype=torch.bfloat16, device="cuda")
        y16 = torch.empty_like(x16)
        torch.cuda.synchronize()
        def calls():
            n.softmax(x16, y16, acsr[4], acsr[5])
            n.sddmm(qd, kt, s, acsr[2], acsr[3], acsr[4], acsr[5])
            n.softmax(s, p, acsr[4], acsr[5], 0.125)
            n.spmm(p, vd, o, acsr[2], acsr[3], acsr[4], acsr[5])
        meta = ao.metadata_from_pattern(ao.PATTERN_CAUSAL_WINDOWED, L, 40, 0, 16)
        for attempt in ("first calls", "known metadata"):
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                calls()
            o.fill_(float("nan")); y16.fill_(float("nan"))
            g.replay()
            torch.cuda.synchronize()
            assert_close(o, at.attention_acsr(q, k.transpose(2, 3), v, meta, acsr[5], 0.125), torch.float32, attempt)
            assert_close(y16, at.softmax_acsr(x16.cpu(), meta), torch.bfloat16, attempt)
            calls()
            torch.cuda.synchronize()
        """)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("shape", ["flat", "one batch", "slices"])
def test_forward_host_takes_any_split_of_batch_and_heads(shape):
    """Operands that view as (1, batch * heads, L, d), whatever their own leading dimensions; others are refused."""
    import acsr_helpers as ah
    import r_attention
    B, H, L, d = 2, 3, 256, 64
    attn = r_attention.RegularAttention(B, L, H, d, ah.create_causal_windowed_mask(L, 30), 16, 16, 0, torch.bfloat16)
    torch.manual_seed(5)
    q, k, v = (torch.randn(B, H, L, d).to(torch.bfloat16) for _ in range(3))
    out = torch.empty_like(q).pin_memory()
    attn.forward_host(q.pin_memory(), k.pin_memory(), v.pin_memory(), out)
    torch.cuda.synchronize()
    if shape == "slices":           # rows of a wider array, also for the result
        wide = [torch.zeros(B, H, L, 2 * d, dtype=torch.bfloat16).pin_memory() for _ in range(4)]
        operands = [t[..., :d] for t in wide]
        for t, x in zip(operands, (q, k, v)):
            t.copy_(x)
        other = operands[3]
    else:
        other = torch.empty((B * H, L, d) if shape == "flat" else (1, B * H, L, d), dtype=torch.bfloat16).pin_memory()
        operands = [q.pin_memory(), k.view(other.shape).pin_memory(), v.view(other.shape).pin_memory(), other]
    result = attn.forward_host(*operands)
    torch.cuda.synchronize()
    assert result is other and torch.equal(other.reshape(out.shape), out)
    with pytest.raises(RuntimeError):
        attn.forward_host(q, k.transpose(1, 2), v, out)
    with pytest.raises(RuntimeError):
        attn.forward_host(q, k[:, :, 1:], v, out)


@pytest.mark.parametrize("call", ["attn([x, x.transpose(2, 3), x])", "n.spmm(s, x, o, *meta, T); n.spmm(s, x, o, *meta, T)",
                                  "n.sddmm(x, x.transpose(2, 3), s, *meta, T); n.sddmm(x, x.transpose(2, 3), s, *meta, T)"])
def test_cuda_core_warning_as_an_error(call):
    """A caller who turns warnings into errors gets one for 16-bit operands on the CUDA cores."""
    r = run_python(f"""
        import acsr_helpers as ah, r_attention, splat_native as n, warnings
        mask = torch.zeros(64, 64, dtype=torch.uint8, device="cuda")
        mask[::2, ::2] = 1; mask[1::2, ::3] = 1                # rows of two strides
        attn = r_attention.RegularAttention(1, 64, 1, 64, mask, 16, 16, 0, torch.float16)
        T, meta = attn.acsr_trailing_dim, (attn.sTod_linear_transformations, attn.sTod_translations, attn.nnzs)
        x = torch.randn(1, 1, 64, 64, dtype=torch.float16, device="cuda")
        s, o = torch.zeros(1, 1, 64, T, dtype=torch.float16, device="cuda"), torch.empty_like(x)
        warnings.simplefilter("error")
        try:
            {call}
        except RuntimeWarning:
            print("raised")
        """)
    assert r.returncode == 0 and "raised" in r.stdout, (r.stdout, r.stderr[-2000:])


def test_only_calls_that_read_it_make_the_band_table():
    import acsr_helpers as ah
    import splat_native as n
    L, d = 256, 64
    for dtype in (torch.float32, torch.bfloat16):
        acsr = ah.create_acsr(ah.create_causal_windowed_mask(L, 40), 16, 0)
        q = torch.randn(1, 2, L, d, device="cuda").to(dtype)
        s, o = torch.empty(1, 2, L, acsr[5], dtype=dtype, device="cuda"), torch.empty_like(q)
        for _ in range(2):
            n.sddmm(q, q.transpose(2, 3), s, acsr[2], acsr[3], acsr[4], acsr[5])
            n.spmm(s, q, o, acsr[2], acsr[3], acsr[4], acsr[5])
            n.attention_fused(q, q.transpose(2, 3), q, o, acsr[2], acsr[3], acsr[4])
        table = acsr[4]._splat_plan[4]
        assert (table is None) if dtype == torch.float32 else table.numel() == 2 * (L + 2)


@pytest.mark.parametrize("call", ["module", "sddmm", "host"])
def test_first_calls_on_two_streams(call):
    """The band table is made on one stream, behind work that is queued there; a call on another one reads it whole."""
    import acsr_helpers as ah
    import r_attention
    import splat_native as n
    L, H, d, dtype = 640, 2, 64, torch.bfloat16
    one, other = torch.cuda.Stream(), torch.cuda.Stream()
    q, k, v = (torch.randn(1, H, L, d, device="cuda").to(dtype) for _ in range(3))
    hosts = [t.cpu().pin_memory() for t in (q, k, v)]

    def make():
        return r_attention.RegularAttention(1, L, H, d, ah.create_causal_windowed_mask(L, 200), 16, 16, 0, dtype, scale=0.125)

    def run(attn):
        if call == "module":
            return attn([q, k.transpose(2, 3), v])
        if call == "host":
            return attn.forward_host(*hosts, torch.empty(1, H, L, d, dtype=dtype).pin_memory())
        s = torch.full((1, H, L, attn.acsr_trailing_dim), float("nan"), dtype=dtype, device="cuda")
        n.sddmm(q, k.transpose(2, 3), s, attn.sTod_linear_transformations, attn.sTod_translations, attn.nnzs, attn.acsr_trailing_dim)
        return s

    expected = run(make()).clone()
    torch.cuda.synchronize()
    attn = make()
    meta = attn.sTod_linear_transformations, attn.sTod_translations, attn.nnzs
    attn.nnzs._splat_plan = attn.nnzs._splat_plan[:4] + (None, 0)         # as classify() leaves it
    torch.cuda.synchronize()
    with torch.cuda.stream(one):
        torch.cuda._sleep(400_000_000)         # SM clocks, some 0.2 s
        n.band_table(*meta, L)
    with torch.cuda.stream(other):
        first, second = run(attn).clone(), run(attn)
    other.synchronize()
    torch.cuda.synchronize()
    if call != "host":                         # (the copy of a host result does not wait for it)
        assert torch.equal(first, expected)
    assert torch.equal(second, expected)
