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
