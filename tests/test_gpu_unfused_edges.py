"""GPU: the 16-byte-piece SDDMM and SpMM and the register softmax at the sizes where pieces, steps and rows do not
line up: trailing dimensions of every remainder, classes of unequal length, head dimensions below a tile's
width, sparse arrays that begin inside a piece, rows longer and shorter than a lane's pieces."""
import pytest
import torch

from conftest import assert_close
from oracle import acsr_oracle as ao
from oracle import attention_oracle as at

pytestmark = pytest.mark.gpu

#        kind, L, p0, p1
PATTERNS = [
    (ao.PATTERN_CAUSAL_WINDOWED, 520, 255, 0),    # rows of 256: whole pieces
    (ao.PATTERN_CAUSAL_WINDOWED, 300, 64, 0),     # 65
    (ao.PATTERN_WINDOWED, 333, 30, 0),            # 61
    (ao.PATTERN_CAUSAL_WINDOWED, 130, 2, 0),      # 3: every piece shared by rows
    (ao.PATTERN_BLOCKED, 200, 37, 0),             # 74
    (ao.PATTERN_STRIDED, 1003, 7, 0),             # classes of 144 and 143 rows, single-element rows
    (ao.PATTERN_DILATED, 769, 300, 3),            # classes of 257, 256, 256 rows
    (ao.PATTERN_CAUSAL_WINDOWED, 256, 0, 0),      # single-element rows only
]


def _shifted(shape, dtype, lead):
    """A contiguous tensor that begins `lead` elements into its allocation."""
    n = 1
    for x in shape:
        n *= x
    return torch.full((n + 16,), float("nan"), dtype=dtype, device="cuda")[lead:lead + n].view(shape)


@pytest.mark.parametrize("lead", [0, 3])
@pytest.mark.parametrize("d", [32, 64, 104, 128])
def test_sddmm_and_spmm_pieces(d, lead):
    import acsr_helpers as ah
    import splat_native as n
    dtype, H = (torch.bfloat16 if d % 64 else torch.float16), 2
    for i, (kind, L, p0, p1) in enumerate(PATTERNS):
        torch.manual_seed(60 + i)
        acsr = ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0)
        meta = ao.metadata_from_pattern(kind, L, p0, p1, 16)
        T, what = acsr[5], f"{(kind, L, p0, p1)} d={d} lead={lead}"
        q, k, v = (torch.randn(1, H, L, d).to(dtype) for _ in range(3))
        s = _shifted((1, H, L, T), dtype, lead)
        n.sddmm(q.cuda(), k.cuda().transpose(2, 3), s, acsr[2], acsr[3], acsr[4], T, n.PATH_BAND)
        assert_close(s, at.sddmm_acsr(q, k.transpose(2, 3), meta, T), dtype, f"sddmm {what}")
        _cols, valid = at._cols(meta, T)
        assert torch.count_nonzero(s.cpu().float() * (~valid)) == 0, "padding slots must be zero"
        p = torch.rand(1, H, L, T)
        p_dev = _shifted((1, H, L, T), dtype, lead)
        p_dev.copy_(torch.where(valid, p, torch.full_like(p, float("nan"))))     # padding is not read
        o = torch.full((1, H, L, d), float("nan"), dtype=dtype, device="cuda")
        n.spmm(p_dev, v.cuda(), o, acsr[2], acsr[3], acsr[4], T, n.PATH_BAND)
        n.check_status_word(0)
        assert_close(o, at.spmm_acsr(p.to(dtype), v, meta), dtype, f"spmm {what}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("lead", [0, 1])
def test_softmax_row_lengths(dtype, lead):
    """One to sixteen pieces per lane and beyond, rows that begin anywhere in a piece, clipped and empty rows,
    negative and zero scales, in place."""
    import splat_native as n
    v = 4 if dtype == torch.float32 else 8
    for T in (1, 5, v, 32 * v - 1, 32 * v, 32 * v + 1, 64 * v, 95 * v + 3, 127 * v, 200 * v + 1, 511 * v, 513 * v + 2):
        L = 37
        torch.manual_seed(T)
        nnz = torch.randint(0, T + 1, (L,))
        nnz[0], nnz[1] = T, 0
        x = (torch.randn(1, 2, L, T) * 3).to(dtype)
        valid = torch.arange(T)[None, :] < nnz[:, None]
        for scale in (0.7, -0.4, 0.0):
            ref = torch.softmax(torch.where(valid, x.float() * scale, torch.tensor(-torch.inf)), -1).nan_to_num(0.0)
            xd = _shifted((1, 2, L, T), dtype, lead)
            xd.copy_(torch.where(valid, x, torch.full_like(x, float("nan"))))     # padding is not read
            n.softmax(xd, xd, nnz.float().cuda(), T, scale)
            assert_close(xd, ref, dtype, f"softmax T={T} scale={scale}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_softmax_lanes_per_row(dtype):
    """Both sides of every change in how many lanes and warps share a row; fewer rows than a block takes, and more."""
    import splat_native as n
    v = 4 if dtype == torch.float32 else 8
    for pieces in (8, 16, 24, 32, 40, 64, 80, 96, 128, 160, 192, 256, 384, 512, 768, 1024, 2048):
        for T, L in ((pieces * v, 3), (pieces * v, 131), (pieces * v + 1, 5)):
            torch.manual_seed(T + L)
            nnz = torch.randint(0, T + 1, (L,))
            nnz[0], nnz[1] = T, 0
            x = torch.randn(1, 1, L, T).to(dtype)
            valid = torch.arange(T)[None, :] < nnz[:, None]
            ref = torch.softmax(torch.where(valid, x.float() * 0.7, torch.tensor(-torch.inf)), -1).nan_to_num(0.0)
            out = torch.full((1, 1, L, T), float("nan"), dtype=dtype, device="cuda")
            n.softmax(x.cuda(), out, nnz.float().cuda(), T, 0.7)
            assert_close(out, ref, dtype, f"softmax T={T} L={L}")


@pytest.mark.parametrize("d", [64, 32])
@pytest.mark.parametrize("lead", [0, 3])
def test_spmm_more_tiles_than_fit_twice(d, lead):
    """SpMM with more than two 128-row tiles per SM (296 on 148), which run three to an SM with a shorter pipeline."""
    import acsr_helpers as ah
    import splat_native as n
    for kind, L, p0, p1, H in ((ao.PATTERN_CAUSAL_WINDOWED, 300, 256, 0, 99), (ao.PATTERN_WINDOWED, 700, 130, 0, 50),
                               (ao.PATTERN_STRIDED, 1003, 7, 0, 22)):
        torch.manual_seed(L + d)
        acsr = ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0)
        meta = ao.metadata_from_pattern(kind, L, p0, p1, 16)
        T = acsr[5]
        v = torch.randn(1, H, L, d).half()
        _cols, valid = at._cols(meta, T)
        p = torch.rand(1, H, L, T)
        p_dev = _shifted((1, H, L, T), torch.float16, lead)
        p_dev.copy_(torch.where(valid, p, torch.full_like(p, float("nan"))))     # padding is not read
        o = torch.full((1, H, L, d), float("nan"), dtype=torch.float16, device="cuda")
        n.spmm(p_dev, v.cuda(), o, acsr[2], acsr[3], acsr[4], T, n.PATH_BAND)
        n.check_status_word(0)
        assert_close(o, at.spmm_acsr(p.half(), v, meta), torch.float16, f"spmm {(kind, L, p0, p1, H)} d={d} lead={lead}")
