"""GPU: a row's result depends on the row's own keys alone.  Q, K and V rows outside a row's band may hold anything --
padding that was never written, infinities -- and what is not finite inside the band shows in the result."""
import pytest
import torch

from oracle import acsr_oracle as ao
from oracle import attention_oracle as at

pytestmark = pytest.mark.gpu

#        kind, L, p0, p1, heads
PATTERNS = [
    (ao.PATTERN_CAUSAL_WINDOWED, 300, 299, 0, 2),     # dense causal; row 0 has one key
    (ao.PATTERN_CAUSAL_WINDOWED, 640, 63, 0, 2),
    (ao.PATTERN_CAUSAL_WINDOWED, 640, 15, 0, 50),     # 64-row fp32 tiles
    (ao.PATTERN_BLOCKED, 400, 96, 0, 2),
    (ao.PATTERN_DILATED, 301, 90, 3, 2),              # classes of unequal length
    (ao.PATTERN_STRIDED, 60, 40, 0, 2),               # rows with one key and rows with two
]
FORMS = [(torch.float32, 64), (torch.float32, 32), (torch.float32, 128), (torch.bfloat16, 64), (torch.bfloat16, 128),
         (torch.float16, 32)]
NAN, INF = float("nan"), float("inf")


def _spoil(t):
    """A NaN and an infinity of either sign in four rows of (1, H, L, d)."""
    L = t.shape[2]
    for i, r in enumerate((0, L // 3, L // 2 + 1, L - 1)):
        t[:, :, r, 3 * i] = (NAN, INF, -INF, NAN)[i]
    return t


def _spmm(p, v, meta):
    """sum over a row's own slots (the oracle multiplies padding slots by V[0])"""
    cols, valid = at._cols(meta, p.shape[3])
    out = torch.zeros(v.shape)
    for j in range(p.shape[3]):
        out += torch.where(valid[:, j, None], p[:, :, :, j, None].float() * v[:, :, cols[:, j]].float(), torch.zeros(()))
    return out


def _attention(q, k, v, meta, T, scale):
    s = at.sddmm_acsr(q, k.transpose(2, 3), meta, T)
    valid = at._cols(meta, T)[1]
    return _spmm(torch.softmax(torch.where(valid, s * scale, torch.tensor(-INF)), -1), v, meta)


def _same(out, ref, dtype, what):
    out = out.float().cpu()
    finite = torch.isfinite(ref)
    wrong = torch.isfinite(out) != finite
    assert not wrong.any(), f"{what}: {int(wrong.sum())} of {wrong.numel()}, first {torch.nonzero(wrong)[0].tolist()}"
    a, r = out[finite], ref[finite]
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    assert ((a - r).abs() <= tol + tol * r.abs()).all(), what


@pytest.mark.parametrize("spoilt", ["v", "k", "q"])
@pytest.mark.parametrize("dtype,d", FORMS)
def test_fused_rows_keep_to_their_keys(dtype, d, spoilt):
    import acsr_helpers as ah
    import splat_native as n
    for i, (kind, L, p0, p1, H) in enumerate(PATTERNS):
        if dtype != torch.float32 and d in (64, 128) and kind not in (ao.PATTERN_DILATED, ao.PATTERN_STRIDED):
            continue        # classes of one length: the fused kernels ask for finite V (splat_b200.h)
        acsr = ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0)
        meta = ao.metadata_from_pattern(kind, L, p0, p1, 16)
        torch.manual_seed(60 + i)
        x = {name: torch.randn(1, H, L, d).to(dtype) for name in "qkv"}
        _spoil(x[spoilt])
        q, k, v = x["q"], x["k"], x["v"]
        for contiguous in (False, True):
            kt = k.cuda().transpose(2, 3)
            out = torch.full((1, H, L, d), 5.0, dtype=dtype, device="cuda")
            n.attention_fused(q.cuda(), kt.contiguous() if contiguous else kt, v.cuda(), out, acsr[2], acsr[3], acsr[4],
                              d ** -0.5)
            _same(out, _attention(q, k, v, meta, acsr[5], d ** -0.5), dtype, f"{(kind, L, p0, p1, H)} {contiguous}")


@pytest.mark.parametrize("dtype,d", FORMS)
def test_spmm_rows_keep_to_their_keys(dtype, d):
    import acsr_helpers as ah
    import splat_native as n
    for i, (kind, L, p0, p1, H) in enumerate(PATTERNS):
        acsr = ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0)
        meta = ao.metadata_from_pattern(kind, L, p0, p1, 16)
        torch.manual_seed(80 + i)
        p = torch.rand(1, H, L, acsr[5]).to(dtype)
        v = _spoil(torch.randn(1, H, L, d).to(dtype))
        out = torch.full((1, H, L, d), 5.0, dtype=dtype, device="cuda")
        n.spmm(p.cuda(), v.cuda(), out, acsr[2], acsr[3], acsr[4], acsr[5])
        _same(out, _spmm(p, v, meta), dtype, f"{(kind, L, p0, p1, H)}")


@pytest.mark.parametrize("dtype,d", [(torch.float32, 64), (torch.float16, 32)])
def test_rows_without_a_finite_score(dtype, d):
    """Every score of some rows minus infinity: no distribution, NaN as a softmax gives it."""
    import acsr_helpers as ah
    import splat_native as n
    L, H, p0 = 200, 2, 9
    acsr = ah.create_acsr(ah.create_causal_windowed_mask(L, p0), 16, 0)
    q, k, v = (torch.ones(1, H, L, d).to(dtype) for _ in range(3))
    k[:, :, 50:90, 0] = -INF                      # rows 59 .. 89 see nothing else
    out = torch.full((1, H, L, d), 5.0, dtype=dtype, device="cuda")
    n.attention_fused(q.cuda(), k.cuda().transpose(2, 3), v.cuda(), out, acsr[2], acsr[3], acsr[4], 1.0)
    none = torch.zeros(L, dtype=torch.bool)
    none[50 + p0:90] = True
    out = out.cpu()
    assert torch.isnan(out[:, :, none]).all() and (out[:, :, ~none] - 1).abs().max() < 1e-3


#        dtype, d, heads: fp32 on register tiles, and enough of them, or d = 128, for the tensor cores
LSE_FORMS = [(torch.float32, 32, 2), (torch.float32, 64, 2), (torch.float32, 32, 30), (torch.float32, 64, 30), (torch.float32, 128, 2),
             (torch.float16, 32, 2)]


@pytest.mark.parametrize("dtype,d,H", LSE_FORMS)
def test_log_sum_exp_beside_scores_of_minus_infinity(dtype, d, H):
    """A key whose score is minus infinity has no weight: output and log-sum-exp are those of the row's other keys."""
    import acsr_helpers as ah
    import splat_native as n
    L = 300
    for kind, p0, p1 in ((ao.PATTERN_WINDOWED, 20, 0), (ao.PATTERN_DILATED, 40, 3)):
        acsr = ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0)
        meta = ao.metadata_from_pattern(kind, L, p0, p1, 16)
        torch.manual_seed(d + H)
        q, k, v = (torch.randn(1, H, L, d) for _ in range(3))
        q[:, :, :, 3] = q[:, :, :, 3].abs() + 0.1
        k[:, :, 50, 3] = k[:, :, 200, 3] = -INF
        if dtype == torch.float32:
            k[:, :, 120, 3] = -3.395e38                  # infinite in bf16
        q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
        scale = d ** -0.5
        scores = at.sddmm_acsr(q, k.transpose(2, 3), meta, acsr[5])
        ref_o, ref_lse = _attention(q, k, v, meta, acsr[5], scale), at.lse_acsr(scores, meta, scale)
        assert torch.isfinite(ref_o).all() and torch.isinf(scores).any()
        for contiguous in (False, True):
            kt = k.cuda().transpose(2, 3)
            out = torch.full((1, H, L, d), 5.0, dtype=dtype, device="cuda")
            lse = torch.full((1, H, L), 5.0, device="cuda")
            n.attention_fused(q.cuda(), kt.contiguous() if contiguous else kt, v.cuda(), out, acsr[2], acsr[3], acsr[4], scale, lse=lse)
            n.check_status_word(0)
            _same(out, ref_o, dtype, f"{kind} {contiguous}")
            _same(lse, ref_lse, torch.float32, f"lse {kind} {contiguous}")
