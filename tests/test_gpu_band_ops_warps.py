"""GPU: 16-bit SDDMM and SpMM with one and with two warps to 32 rows.  A row's result does not depend on which it is, so a few
heads alone (always two) have the bits that they have among many (one, where rows are long)."""
import pytest
import torch

import acsr_helpers as ah
import splat_native as n

pytestmark = pytest.mark.gpu

#        mask, L, heads: rows of more than 512 non-zeros, more than 296 tiles together
PATTERNS = [
    (lambda L: ah.create_causal_windowed_mask(L, L - 1), 645, 60),        # rows of every length; row 0 has one key
    (lambda L: ah.create_windowed_mask(L, 300), 1027, 40),                # rows begin at any element
    (lambda L: ah.create_blocked_mask(L, 300), 1000, 40),
    (lambda L: ah.create_dilated_mask(L, 600, 2), 1300, 35),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [40, 64, 128])
def test_few_heads_have_the_bits_of_many(d, dtype):
    for mask, L, H in PATTERNS:
        acsr = ah.create_acsr(mask(L), 16, 0)
        meta, T = acsr[2:5], acsr[5]
        assert T > 512
        g = torch.Generator(device="cuda").manual_seed(L + d)
        q, k, v = (torch.empty(1, H, L, d, dtype=dtype, device="cuda").normal_(generator=g) for _ in range(3))
        s, o = torch.full((1, H, L, T), float("nan"), dtype=dtype, device="cuda"), torch.full_like(q, float("nan"))
        n.sddmm(q, k.transpose(2, 3), s, *meta, T, n.PATH_BAND)
        p = torch.empty_like(s)
        n.softmax(s, p, acsr[4], T, d ** -0.5)
        n.spmm(p, v, o, *meta, T, n.PATH_BAND)
        assert torch.isfinite(s.float()).all() and torch.isfinite(o.float()).all()
        for h in (0, H - 1):
            one = slice(h, h + 1)
            s1, o1 = torch.full((1, 1, L, T), float("nan"), dtype=dtype, device="cuda"), torch.full_like(q[:, one], float("nan"))
            n.sddmm(q[:, one], k[:, one].transpose(2, 3), s1, *meta, T, n.PATH_BAND)
            n.spmm(p[:, one].contiguous(), v[:, one], o1, *meta, T, n.PATH_BAND)
            assert torch.equal(s1, s[:, one]) and torch.equal(o1, o[:, one]), (L, h)
    n.check_status_word(0)
