"""GPU: the fp32 register-tile kernels (fused, SDDMM, SpMM) against the CPU oracle at the edges of their
tiles: lengths around multiples of 64, classes with a missing last row, both K layouts, rows with one or
no non-zero.  Without a status word the library runs them at any size; the launchers, which have one, hand what is more than
a wave or two of their tiles to the tensor cores (test_gpu_split_f32.py)."""
import ctypes

import pytest
import torch

from conftest import assert_close
from oracle import acsr_oracle as ao
from oracle import attention_oracle as at

pytestmark = pytest.mark.gpu

#        kind, L, p0, p1, heads (64-row CTAs from 444 of them over all heads, below that 32-row ones of four warps from 296,
#        else of eight)
PATTERNS = [
    (ao.PATTERN_CAUSAL_WINDOWED, 65, 63, 0, 3),      # one row in the second tile
    (ao.PATTERN_CAUSAL_WINDOWED, 127, 126, 0, 3),    # dense causal, one row short of two tiles
    (ao.PATTERN_CAUSAL_WINDOWED, 389, 64, 0, 64),    # L not a multiple of 4; 448 tiles
    (ao.PATTERN_WINDOWED, 256, 37, 0, 111),          # 444 tiles
    (ao.PATTERN_BLOCKED, 200, 48, 0, 3),
    (ao.PATTERN_BLOCKED, 200, 48, 0, 50),            # 350 32-row tiles, 200 64-row ones
    (ao.PATTERN_STRIDED, 203, 8, 0, 56),             # classes of 26 and 25 rows, single-element rows; 448 tiles
    (ao.PATTERN_DILATED, 301, 40, 3, 3),             # classes of 101 and 100 rows
    (ao.PATTERN_CAUSAL_WINDOWED, 3, 1, 0, 3),        # smallest
]


def _tiles(plan, L, H):
    """Tiles of 32 rows."""
    stride = plan[1] if plan[7] > 0 else 1
    return -(-(-(-L // stride)) // 32) * stride * H


class _Tiles:
    """The three operators on the register tiles: the library's entry points without a status word."""

    def __init__(self, acsr, L, H, d):
        import splat_native as n
        self.n, self.T, self.sizes = n, acsr[5], (H, L, L, d)
        self.plan = n.classify(acsr[2], acsr[3], acsr[4])
        assert self.plan[3] == 0 and (self.plan[7] == 0 or self.plan[1] == self.plan[2])     # a band pattern
        self.plan_arr = ctypes.cast((ctypes.c_int32 * 8)(*self.plan), ctypes.c_void_p)
        self.acsr, self.vectors = acsr, [t.data_ptr() for t in acsr[2:5]]
        self.fp32 = n.dtype_code(torch.float32)

    def fused(self, q, kt, v, o, lse, scale):
        _bh, ksb, ksk, ksc = self.n._flat_bh(kt, "kt")
        return self.n._lib.splat_attention_fused_table(
            q.data_ptr(), kt.data_ptr(), ksb, ksc, ksk, v.data_ptr(), o.data_ptr(), lse.data_ptr(), *self.vectors, *self.sizes, scale,
            self.fp32, self.n.PATH_AUTO, self.plan_arr, None, None, None, self.n._stream(q.device))

    def sddmm(self, q, kt, s):
        _bh, ksb, ksk, ksc = self.n._flat_bh(kt, "kt")
        return self.n._lib.splat_sddmm_tile(q.data_ptr(), kt.data_ptr(), ksb, ksc, ksk, s.data_ptr(), *self.vectors, *self.sizes, self.T,
                                            self.fp32, self.plan_arr, self.n._stream(q.device))

    def spmm(self, p, v, o):
        return self.n._lib.splat_spmm_tile(p.data_ptr(), v.data_ptr(), o.data_ptr(), *self.vectors, *self.sizes, self.T, self.fp32,
                                           self.plan_arr, self.n._stream(p.device))


@pytest.mark.parametrize("contiguous", [False, True])
@pytest.mark.parametrize("d", [32, 64, 128])
def test_tile_kernels_against_oracle(d, contiguous):
    import acsr_helpers as ah
    import splat_native as n
    for i, (kind, L, p0, p1, H) in enumerate(PATTERNS):
        torch.manual_seed(700 + i)
        acsr = ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0)
        meta = ao.metadata_from_pattern(kind, L, p0, p1, 16)
        T, what = acsr[5], f"{(kind, L, p0, p1)} d={d}"
        q, k, v = (torch.randn(1, H, L, d) for _ in range(3))
        qd, kt, vd = q.cuda(), k.cuda().transpose(2, 3), v.cuda()
        kt = kt.contiguous() if contiguous else kt
        scale = d ** -0.5
        tile, tiles = _Tiles(acsr, L, H, d), _tiles(n.classify(*acsr[2:5]), L, H)
        s_ref = at.sddmm_acsr(q, k.transpose(2, 3), meta, T)
        _cols, valid = at._cols(meta, T)
        p = torch.rand(1, H, L, T)
        p_dev = torch.where(valid, p, torch.full_like(p, float("nan"))).cuda()     # padding is not read
        nan = lambda *shape: torch.full(shape, float("nan"), device="cuda")
        o, lse, s, o2 = nan(1, H, L, d), nan(1, H, L), nan(1, H, L, T), nan(1, H, L, d)
        assert tile.fused(qd, kt, vd, o, lse, scale) == 0 and tile.sddmm(qd, kt, s) == 0, what
        assert_close(o, at.attention_acsr(q, k.transpose(2, 3), v, meta, T, scale), torch.float32, f"fused {what}")
        assert_close(lse, at.lse_acsr(s_ref, meta, scale), torch.float32, f"lse {what}")
        assert_close(s, s_ref, torch.float32, f"sddmm {what}")
        assert torch.count_nonzero(s.cpu() * (~valid)) == 0, "padding slots must be zero"
        if L > 32:      # (row kernels sum in another order)
            rows = torch.empty_like(o)
            n.attention_fused(qd, kt, vd, rows, acsr[2], acsr[3], acsr[4], scale, n.PATH_GENERIC)
            assert not torch.equal(o, rows), f"fused {what}: the row kernel"
        rc = tile.spmm(p_dev, vd, o2)
        if kind == ao.PATTERN_STRIDED:      # classes of 26 rows: too short for SpMM, which the row kernel does
            assert rc == n.ERR_UNSUPPORTED_SHAPE
        else:
            assert rc == 0
            assert_close(o2, at.spmm_acsr(p, v, meta), torch.float32, f"spmm {what}")
        # the launchers: the same kernels, so the same bits, up to the lines behind which the tensor cores take over
        lo, ls, lo2 = nan(1, H, L, d), nan(1, H, L, T), nan(1, H, L, d)
        n.attention_fused(qd, kt, vd, lo, acsr[2], acsr[3], acsr[4], scale, n.PATH_AUTO)
        n.sddmm(qd, kt, ls, acsr[2], acsr[3], acsr[4], T)
        n.spmm(p_dev, vd, lo2, acsr[2], acsr[3], acsr[4], T)
        assert_close(ls, s_ref, torch.float32, f"sddmm launcher {what}")
        assert_close(lo2, at.spmm_acsr(p, v, meta), torch.float32, f"spmm launcher {what}")
        if tiles <= 148 and d < 128:
            assert torch.equal(lo, o), what
        if tiles <= (296 if d == 32 else 148):
            assert torch.equal(ls, s), what
        if rc == 0 and tiles <= (148 if d == 128 else 296):
            assert torch.equal(lo2, o2), what


@pytest.mark.parametrize("d", [32, 64])
def test_sddmm_and_spmm_on_either_side_of_each_register_budget(d):
    """CTAs of eight warps up to 148 and from there, of 32 and of 64 rows up to 470, to 614, to 888 and from there."""
    import acsr_helpers as ah
    for L, H in [(64, 74), (64, 75), (96, 156), (96, 157), (96, 204), (96, 205), (64, 470), (64, 471), (64, 614), (64, 615), (64, 888),
                 (64, 889)]:
        acsr = ah.create_acsr(ah.create_windowed_mask(L, 21), 16, 0)
        meta = ao.metadata_from_pattern(ao.PATTERN_WINDOWED, L, 21, 0, 16)
        T = acsr[5]
        g = torch.Generator(device="cuda").manual_seed(L + H)
        q, k, v = (torch.randn(1, H, L, d, device="cuda", generator=g) for _ in range(3))
        s, o = torch.full((1, H, L, T), float("nan"), device="cuda"), torch.full_like(q, float("nan"))
        tile = _Tiles(acsr, L, H, d)
        assert tile.sddmm(q, k.transpose(2, 3), s) == 0 and tile.spmm(s, v, o) == 0
        assert_close(s, at.sddmm_acsr(q.cpu(), k.cpu().transpose(2, 3), meta, T), torch.float32, f"sddmm {L} {H}")
        # sums of 43 products of normal values: 2^-24 of some 43 sqrt(d) each, well under the tolerance
        assert_close(o / d ** 0.5, at.spmm_acsr(s.cpu(), v.cpu(), meta) / d ** 0.5, torch.float32, f"spmm {L} {H}")
