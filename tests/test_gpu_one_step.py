"""GPU: the fused 16-bit kernel of classes with up to 64 rows (one step of 64 keys, d <= 64) on either side of its edge,
against the CPU oracle; rows with one key and with none, classes of unequal length, both K layouts, the log-sum-exp."""
import numpy as np
import pytest
import torch

import acsr_helpers as ah
import splat_native as n
from conftest import assert_close
from oracle import acsr_oracle as ao
from oracle import attention_oracle as at

pytestmark = pytest.mark.gpu

#        kind, L, p0, p1: rows of a class
PATTERNS = [
    (ao.PATTERN_CAUSAL_WINDOWED, 1, 0, 0),         # one
    (ao.PATTERN_CAUSAL_WINDOWED, 40, 7, 0),
    (ao.PATTERN_WINDOWED, 64, 20, 0),              # 64
    (ao.PATTERN_WINDOWED, 65, 20, 0),              # 65: the kernel with 128-key steps
    (ao.PATTERN_BLOCKED, 56, 16, 0),
    (ao.PATTERN_STRIDED, 512, 8, 0),               # 64
    (ao.PATTERN_STRIDED, 508, 8, 0),               # 64 and 63
    (ao.PATTERN_STRIDED, 513, 8, 0),               # 65 and 64
    (ao.PATTERN_STRIDED, 100, 60, 0),              # 2 and 1
    (ao.PATTERN_DILATED, 250, 9, 4),               # 63 and 62
    ("ragged", 61, 0, 0),
    ("ragged", 64, 0, 0),
    ("ragged", 130, 0, 0),                         # 130: 128-key steps
]


def ragged_mask(L):
    """Windows of every length, rows with one key (the metadata have it as column 0) and rows with none."""
    g = np.random.default_rng(L)
    row = np.arange(L)
    lo, hi = np.maximum(row - g.integers(0, 12, L), 0), row + g.integers(0, 9, L)
    mask = ((row[None] >= lo[:, None]) & (row[None] <= hi[:, None])).astype(np.uint8)
    mask[::7] = 0
    mask[3::11] = row[None] == row[3::11, None]
    return mask


def case(kind, L, p0, p1):
    """(device metadata, the oracle's); kind "ragged": an explicit mask."""
    if kind != "ragged":
        return ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0), ao.metadata_from_pattern(kind, L, p0, p1, 16)
    mask = ragged_mask(L)
    assert (mask.sum(1) == 0).any() and (mask.sum(1) == 1).any()
    return ah.create_acsr(torch.from_numpy(mask).cuda(), 16, 0), ao.metadata_from_mask(mask, 16)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [8, 32, 64])
def test_classes_of_one_step(d, dtype):
    for i, (kind, L, p0, p1) in enumerate(PATTERNS):
        acsr, meta = case(kind, L, p0, p1)
        T, scale, H = acsr[5], d ** -0.5, 3
        torch.manual_seed(900 + i)
        q, k, v = (torch.randn(1, H, L, d).to(dtype) for _ in range(3))
        ref = at.attention_acsr(q, k.transpose(2, 3), v, meta, T, scale)
        ref_lse = at.lse_acsr(at.sddmm_acsr(q, k.transpose(2, 3), meta, T), meta, scale)
        for contiguous in (False, True):
            kt = k.cuda().transpose(2, 3)
            kt = kt.contiguous() if contiguous else kt
            o = torch.full((1, H, L, d), float("nan"), dtype=dtype, device="cuda")
            lse = torch.full((1, H, L), float("nan"), device="cuda")
            n.attention_fused(q.cuda(), kt, v.cuda(), o, acsr[2], acsr[3], acsr[4], scale, n.PATH_AUTO, lse=lse)
            what = f"{(kind, L, p0, p1)} d={d} contiguous={contiguous}"
            assert_close(o, ref, dtype, what)
            # scores are summed in fp32: 2^-24 of some 8 sqrt(d) terms
            empty = torch.isinf(ref_lse)
            assert torch.equal(lse.cpu()[empty], ref_lse[empty]), f"rows without a key, {what}"
            assert_close(lse.cpu()[~empty], ref_lse[~empty], torch.float32, f"lse {what}")
            plain = torch.full_like(o, float("nan"))
            n.attention_fused(q.cuda(), kt, v.cuda(), plain, acsr[2], acsr[3], acsr[4], scale, n.PATH_AUTO)
            assert torch.equal(o, plain), f"the log-sum-exp output changes the result, {what}"
    n.check_status_word(0)
