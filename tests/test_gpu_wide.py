"""GPU: the 128-key-step band kernel (the default for band patterns) against the CPU oracle, at the sizes
where its steps, chunks and classes can go wrong: bands that begin and end inside a half step or chunk,
single-tile classes, classes of unequal length, head dimensions below a tile's width, ragged lengths, rows
without a band, both K^T layouts, the log-sum-exp output."""
import pytest
import torch

from conftest import assert_close
from oracle import acsr_oracle as ao
from oracle import attention_oracle as at

pytestmark = pytest.mark.gpu

#        kind, L, p0, p1, heads
PATTERNS = [
    (ao.PATTERN_CAUSAL_WINDOWED, 128, 127, 0, 1),     # one tile, one step
    (ao.PATTERN_CAUSAL_WINDOWED, 129, 40, 0, 2),      # one row in the second tile
    (ao.PATTERN_CAUSAL_WINDOWED, 640, 255, 0, 3),     # edge, interior and edge step
    (ao.PATTERN_CAUSAL_WINDOWED, 640, 63, 0, 2),      # half steps at both ends
    (ao.PATTERN_CAUSAL_WINDOWED, 1024, 1023, 0, 2),   # dense causal
    (ao.PATTERN_WINDOWED, 1000, 100, 0, 3),
    (ao.PATTERN_BLOCKED, 512, 96, 0, 2),
    (ao.PATTERN_CAUSAL_WINDOWED, 256, 0, 0, 2),       # single-element rows only: nothing to multiply
    (ao.PATTERN_STRIDED, 512, 4, 0, 2),               # classes of one tile; single-element rows
    (ao.PATTERN_STRIDED, 1024, 64, 0, 2),             # classes of 16 rows
    (ao.PATTERN_STRIDED, 1003, 7, 0, 2),              # two classes of 144 rows, five of 143
    (ao.PATTERN_STRIDED, 60, 64, 0, 2),               # stride > L: single-element rows only
    (ao.PATTERN_DILATED, 1024, 200, 2, 2),            # two classes of four tiles
    (ao.PATTERN_DILATED, 769, 300, 3, 2),             # classes of 257, 256, 256 rows
]


def _run(kind, L, p0, p1, H, d, dtype, seed, contiguous=False, scale=None):
    import acsr_helpers as ah
    import splat_native as n
    torch.manual_seed(seed)
    acsr = ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0)
    meta = ao.metadata_from_pattern(kind, L, p0, p1, 16)
    q, k, v = (torch.randn(1, H, L, d).to(dtype) for _ in range(3))
    scale = d ** -0.5 if scale is None else scale
    kt = k.cuda().transpose(2, 3)
    kt = kt.contiguous() if contiguous else kt
    out = torch.full((1, H, L, d), float("nan"), dtype=dtype, device="cuda")
    lse = torch.full((1, H, L), float("nan"), device="cuda")
    n.attention_fused(q.cuda(), kt, v.cuda(), out, acsr[2], acsr[3], acsr[4], scale, n.PATH_BAND, lse=lse)
    n.check_status_word(0)
    plain = torch.full_like(out, float("nan"))
    n.attention_fused(q.cuda(), kt, v.cuda(), plain, acsr[2], acsr[3], acsr[4], scale, n.PATH_BAND)
    n.check_status_word(0)
    assert torch.equal(out, plain), "the log-sum-exp output changes the result"
    s = at.sddmm_acsr(q, k.transpose(2, 3), meta, meta["trailing_dim"])
    return out, at.attention_acsr(q, k.transpose(2, 3), v, meta, meta["trailing_dim"], scale), lse, at.lse_acsr(s, meta, scale)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [128, 64, 32, 8, 104])
def test_wide_patterns(d, dtype):
    for i, (kind, L, p0, p1, H) in enumerate(PATTERNS):
        for contiguous in (False, True):
            if contiguous and (kind in (ao.PATTERN_STRIDED, ao.PATTERN_DILATED) or L % 8):
                continue
            out, ref, lse, lse_ref = _run(kind, L, p0, p1, H, d, dtype, 900 + i, contiguous)
            what = f"pattern {(kind, L, p0, p1, H)} d={d} contiguous={contiguous}"
            assert_close(out, ref, dtype, what)
            assert (lse.cpu() - lse_ref).abs().max().item() < 2e-2, f"lse, {what}"


def test_wide_unscaled_scores_need_the_running_max():
    """scale = 1 with d = 128 gives scores of sigma ~ 11: exercises the lazy rescale of O."""
    for d in (128, 64):
        out, ref, _lse, _ref = _run(ao.PATTERN_CAUSAL_WINDOWED, 1024, 511, 0, 3, d, torch.bfloat16, 7, scale=1.0)
        assert_close(out, ref, torch.bfloat16, f"unscaled d={d}")
