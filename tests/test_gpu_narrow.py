"""GPU: the fused 16-bit kernels with d up to 32, which read half of a 64-column tile, against the CPU oracle: one, some and many steps,
classes of unequal length, rows with one key and with none, maxima that grow from step to step, both K layouts, the log-sum-exp."""
import pytest
import torch

import acsr_helpers as ah
import splat_native as n
from conftest import assert_close
from oracle import acsr_oracle as ao
from oracle import attention_oracle as at
from test_gpu_one_step import case

pytestmark = pytest.mark.gpu

PATTERNS = [
    (ao.PATTERN_CAUSAL_WINDOWED, 300, 31, 0),
    (ao.PATTERN_WINDOWED, 640, 250, 0),
    (ao.PATTERN_BLOCKED, 400, 96, 0),
    (ao.PATTERN_STRIDED, 333, 3, 0),
    (ao.PATTERN_DILATED, 500, 40, 3),
    ("ragged", 50, 0, 0),
    ("ragged", 390, 0, 0),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [8, 24, 32, 40])
def test_narrow_heads(d, dtype):
    for i, (kind, L, p0, p1) in enumerate(PATTERNS):
        acsr, meta = case(kind, L, p0, p1)
        T, scale, H = acsr[5], d ** -0.5, 2
        torch.manual_seed(40 + i)
        q, k, v = (torch.randn(1, H, L, d).to(dtype) for _ in range(3))
        k = (k.float() * torch.linspace(0.2, 6.0, L)[:, None]).to(dtype)       # later keys have the larger scores
        ref = at.attention_acsr(q, k.transpose(2, 3), v, meta, T, scale)
        ref_lse = at.lse_acsr(at.sddmm_acsr(q, k.transpose(2, 3), meta, T), meta, scale)
        empty = torch.isinf(ref_lse)
        for contiguous in (False, True):
            kt = k.cuda().transpose(2, 3)
            kt = kt.contiguous() if contiguous else kt
            o = torch.full((1, H, L, d), float("nan"), dtype=dtype, device="cuda")
            n.attention_fused(q.cuda(), kt, v.cuda(), o, acsr[2], acsr[3], acsr[4], scale, n.PATH_AUTO)
            assert_close(o, ref, dtype, f"{(kind, L, p0, p1)} d={d} contiguous={contiguous}")
            with_lse, lse = torch.full_like(o, float("nan")), torch.full((1, H, L), float("nan"), device="cuda")
            n.attention_fused(q.cuda(), kt, v.cuda(), with_lse, acsr[2], acsr[3], acsr[4], scale, n.PATH_AUTO, lse=lse)
            assert torch.equal(with_lse, o) and torch.equal(lse.cpu()[empty], ref_lse[empty])
            # scores of up to some 30, summed in fp32: 2^-24 of some 8 sqrt(d) terms
            assert_close(lse.cpu()[~empty], ref_lse[~empty], torch.float32, f"lse {(kind, L, p0, p1)} d={d}")
    n.check_status_word(0)
