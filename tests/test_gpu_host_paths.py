"""GPU: what the launchers do around the kernels -- the one-kernel metadata of an explicit mask, the row-major
copy of a contiguous K^T that the tensor-core kernels cannot fetch, host-resident operands in chunks."""
import numpy as np
import pytest
import torch

from conftest import assert_close, bits_equal
from oracle import acsr_oracle as ao
from oracle import attention_oracle as at

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("height", [4, 16, 64, 3, 65])      # the last two: outside the one-kernel range
@pytest.mark.parametrize("cols", [1, 15, 16, 17, 530, 2200])
def test_metadata_of_ragged_masks(cols, height):
    """Rows of every kind -- affine runs, single elements, none, full -- at widths around the 16-byte loads and
    around a lane's four loads, and at row starts of every alignment (a mask inside a wider array)."""
    import acsr_helpers as ah
    rng = np.random.default_rng(cols)
    rows = 97
    dense = np.zeros((rows, cols), dtype=np.uint8)
    for i in range(rows):
        kind = i % 5
        if kind == 0:
            dense[i, rng.integers(cols)] = 1
        elif kind == 1:
            dense[i, :] = 1
        elif kind >= 3:
            a, step = int(rng.integers(cols)), int(rng.integers(1, 40))
            dense[i, a::step] = 1
    big = torch.zeros(rows, cols + 3, dtype=torch.uint8, device="cuda")
    big[:, 2:2 + cols] = torch.from_numpy(dense)
    ref = ao.metadata_from_mask(dense, height)
    for mask in (torch.from_numpy(dense).cuda(), torch.from_numpy(dense).cuda().bool(), big[:, 2:2 + cols]):
        out = ah.create_acsr(mask, height, 0)
        for i, k in enumerate(("dTos_lin", "dTos_tr", "sTod_lin", "sTod_tr", "nnzs")):
            assert bits_equal(out[i].cpu().numpy(), ref[k]), k
        assert out[5] == ref["trailing_dim"]
        assert bits_equal(out[6].cpu().numpy(), ref["span_start"]) and bits_equal(out[7].cpu().numpy(), ref["span_end"])


@pytest.mark.parametrize("L", [300, 301, 513])
@pytest.mark.parametrize("d", [32, 64, 128])
def test_contiguous_kt_that_is_copied(d, L):
    """Strided and dilated patterns, and lengths that are not a multiple of 8, with the reference's K^T layout."""
    import acsr_helpers as ah
    import r_attention
    import splat_native as n
    for i, (kind, p0, p1) in enumerate([(ao.PATTERN_STRIDED, 5, 0), (ao.PATTERN_DILATED, 60, 2),
                                        (ao.PATTERN_CAUSAL_WINDOWED, 40, 0)]):
        torch.manual_seed(40 + i)
        acsr = ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0)
        meta = ao.metadata_from_pattern(kind, L, p0, p1, 16)
        q, k, v = (torch.randn(2, 3, L, d).to(torch.bfloat16) for _ in range(3))
        kt = k.cuda().transpose(2, 3).contiguous()
        attn = r_attention.RegularAttention(2, L, 3, d, ah.PatternMask(kind, L, p0, p1), 16, 16, 0, torch.bfloat16,
                                            scale=d ** -0.5)
        out = attn([q.cuda(), kt, v.cuda()]).clone()
        # (the kernels on the CUDA cores sum in another order: the same bits mean the same kernel)
        assert torch.equal(out, attn([q.cuda(), k.cuda().transpose(2, 3), v.cuda()])), "not the tensor-core kernel"
        assert_close(out, at.attention_acsr(q, k.transpose(2, 3), v, meta, meta["trailing_dim"], d ** -0.5), torch.bfloat16,
                     f"fused {(kind, L, p0, p1)} d={d}")
        s = torch.full((2, 3, L, acsr[5]), float("nan"), dtype=torch.bfloat16, device="cuda")
        n.sddmm(q.cuda(), kt, s, acsr[2], acsr[3], acsr[4], acsr[5])        # the first call on these metadata
        for other in (kt, k.cuda().transpose(2, 3)):
            again = torch.full_like(s, float("nan"))
            n.sddmm(q.cuda(), other, again, acsr[2], acsr[3], acsr[4], acsr[5])
            assert torch.equal(s, again), f"the first call takes another kernel {(kind, L, p0, p1)} d={d}"
        assert_close(s, at.sddmm_acsr(q, k.transpose(2, 3), meta, acsr[5]), torch.bfloat16, f"sddmm {(kind, L, p0, p1)} d={d}")


def test_contiguous_kt_in_the_python_path(monkeypatch):
    """Calls that the native path leaves to Python (debug mode here) take the kernels that they take without it."""
    import acsr_helpers as ah
    import r_attention
    import splat_native as n
    L, H, d = 301, 2, 64
    attn = r_attention.RegularAttention(1, L, H, d, ah.create_strided_mask(L, 7), 16, 16, 0, torch.float16, scale=0.125)
    q, k, v = (torch.randn(1, H, L, d, device="cuda").half() for _ in range(3))
    x = [q, k.transpose(2, 3).contiguous(), v]
    expected = attn(x).clone()
    monkeypatch.setenv("SPLAT_B200_DEBUG", "1")
    try:
        out = attn(x).clone()
    finally:
        n.check_indices(0, False)
    assert torch.equal(out, expected)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_forward_host_in_chunks(dtype):
    """Several chunks, a last one that is smaller, and a second call on the same staging buffers."""
    import acsr_helpers as ah
    import r_attention
    B, H, L, d = 1, 7, 384, 64
    mask = ah.create_causal_windowed_mask(L, 99)
    meta = ao.metadata_from_pattern(ao.PATTERN_CAUSAL_WINDOWED, L, 99, 0, 16)
    attn = r_attention.RegularAttention(B, L, H, d, mask, 16, 16, 0, dtype, scale=0.125)
    for seed in (1, 2):
        torch.manual_seed(seed)
        q, k, v = (torch.randn(B, H, L, d).to(dtype).pin_memory() for _ in range(3))
        out = torch.full((B, H, L, d), float("nan"), dtype=dtype).pin_memory()
        attn.forward_host(q, k, v, out, chunk_heads=2)
        torch.cuda.current_stream().synchronize()
        assert_close(out, at.attention_acsr(q, k.transpose(2, 3), v, meta, meta["trailing_dim"], 0.125), dtype, f"call {seed}")
    assert [r_attention.host_chunk(h, b) for h, b in ((32, 2 << 20), (6, 400 << 10), (1, 64 << 20), (7, 1 << 20))] == [5, 6, 1, 2]


def test_other_threads_run_while_metadata_wait():
    """create_acsr behind queued work waits without the interpreter lock."""
    import threading
    import time

    import acsr_helpers as ah
    mask = torch.ones(64, 64, dtype=torch.uint8, device="cuda").tril()
    ah.create_acsr(mask, 16, 0)
    took = []

    def metadata():
        t0 = time.monotonic()
        ah.create_acsr(mask, 16, 0)
        took.append(time.monotonic() - t0)
    torch.cuda._sleep(600_000_000)              # SM clocks, some 0.3 s
    thread = threading.Thread(target=metadata)
    thread.start()
    longest, last = 0.0, time.monotonic()
    while thread.is_alive():
        time.sleep(0.001)
        now = time.monotonic()
        longest, last = max(longest, now - last), now
    thread.join()
    assert took[0] > 0.15 and longest < 0.1, (took, longest)


@pytest.mark.parametrize("L", [300, 512])
def test_metadata_of_more_rows_than_the_operands(L):
    """Metadata vectors padded with empty rows: the launchers take vectors of at least L elements."""
    import acsr_helpers as ah
    import splat_native as n
    H, d, dtype = 2, 64, torch.bfloat16
    acsr = ah.create_acsr(ah.create_causal_windowed_mask(L, 40), 16, 0)
    pad = torch.zeros(200, device="cuda")
    lin, tr, nnzs = torch.cat([acsr[2], pad + 1]), torch.cat([acsr[3], pad]), torch.cat([acsr[4], pad])
    meta = ao.metadata_from_pattern(ao.PATTERN_CAUSAL_WINDOWED, L, 40, 0, 16)
    torch.manual_seed(8)
    q, k, v = (torch.randn(1, H, L, d).to(dtype) for _ in range(3))
    qd, kt, vd = q.cuda(), k.cuda().transpose(2, 3), v.cuda()
    p = torch.rand(1, H, L, acsr[5]).to(dtype)
    s, o, fused = torch.empty_like(p, device="cuda"), torch.empty_like(qd), torch.empty_like(qd)
    for _ in range(2):                  # through Python, through the native path
        for t in (s, o, fused):
            t.fill_(float("nan"))
        n.attention_fused(qd, kt, vd, fused, lin, tr, nnzs, 0.125)
        n.sddmm(qd, kt, s, lin, tr, nnzs, acsr[5])
        n.spmm(p.cuda(), vd, o, lin, tr, nnzs, acsr[5])
        assert_close(fused, at.attention_acsr(q, k.transpose(2, 3), v, meta, acsr[5], 0.125), dtype, "fused")
        assert_close(s, at.sddmm_acsr(q, k.transpose(2, 3), meta, acsr[5]), dtype, "sddmm")
        assert_close(o, at.spmm_acsr(p, v, meta), dtype, "spmm")
