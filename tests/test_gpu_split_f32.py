"""GPU: the fp32 kernels on the tensor cores (operands split into three bf16 numbers) at the edges of their tiles of 128 rows
and steps of 64 keys, against 64 bits: with operands of either sign they must not be further off than the kernels that sum with
FMAs."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

import acsr_helpers as ah
import splat_native as n
from conftest import ROOT, SPLAT_DIR

pytestmark = pytest.mark.gpu

#        mask, L, heads (more than 148 tiles of 32 rows together: below, the register tiles run at d = 32 and 64)
PATTERNS = [
    (lambda L: ah.create_causal_windowed_mask(L, L - 1), 128, 38),      # one whole tile
    (lambda L: ah.create_causal_windowed_mask(L, 63), 129, 31),         # one row in the second tile
    (lambda L: ah.create_windowed_mask(L, 3), 70, 50),                  # a tile of 70 rows
    (lambda L: ah.create_windowed_mask(L, 100), 1004, 5),               # K^T in loads of four
    (lambda L: ah.create_windowed_mask(L, 40), 389, 13),                # K^T key by key
    (lambda L: ah.create_blocked_mask(L, 48), 200, 22),
    (lambda L: ah.create_strided_mask(L, 8), 203, 20),                  # classes of 26 and 25 rows, rows with one key
    (lambda L: ah.create_dilated_mask(L, 40, 3), 301, 13),              # classes of 101 and 100 rows
    ("documents", 1000, 5),                                             # ragged bands, rows with one key and with none
]


def _mask(mask, L):
    if mask != "documents":
        return mask(L)
    g = torch.Generator().manual_seed(L)
    row = torch.arange(L)
    lo, hi = (row - torch.randint(0, 90, (L,), generator=g)).clamp(min=0), row + torch.randint(0, 30, (L,), generator=g)
    m = (row[None] >= lo[:, None]) & (row[None] <= hi[:, None])
    m[::17] = False
    m[5::31] = row[None] == row[5::31, None]
    return m.to(torch.uint8).cuda()


def _exact(q, kt, v, acsr, scale):
    """Output and log-sum-exp in 64 bits, from the row metadata."""
    lin, tr, nnz = (t.double() for t in acsr[2:5])
    stride, start = lin.round().clamp(min=1), (lin * tr).round()
    off = torch.arange(q.shape[2], device="cuda").double()[None] - start[:, None]
    on = (off >= 0) & (off < nnz[:, None] * stride[:, None]) & (torch.remainder(off, stride[:, None]) == 0)
    s = (q.double() @ kt.double() * scale).masked_fill(~on, float("-inf"))
    return torch.nan_to_num(torch.softmax(s, -1)) @ v.double(), torch.logsumexp(s, -1)


def _call(q, kt, v, acsr, scale, status=True):
    """(output, log-sum-exp); without a status word the register tiles run."""
    H, L, d = q.shape[1:]
    o, lse = torch.full_like(q, float("nan")), torch.full((1, H, L), float("nan"), device="cuda")
    if status:
        n.attention_fused(q, kt, v, o, acsr[2], acsr[3], acsr[4], scale, lse=lse)
        n.check_status_word(0)
        return o, lse
    plan = (ctypes.c_int32 * 8)(*n.classify(*acsr[2:5]))
    _bh, ksb, ksk, ksc = n._flat_bh(kt, "kt")
    assert n._lib.splat_attention_fused_table(
        q.data_ptr(), kt.data_ptr(), ksb, ksc, ksk, v.data_ptr(), o.data_ptr(), lse.data_ptr(), acsr[2].data_ptr(),
        acsr[3].data_ptr(), acsr[4].data_ptr(), H, L, L, d, scale, n.dtype_code(q.dtype), n.PATH_AUTO,
        ctypes.cast(plan, ctypes.c_void_p), None, None, None, n._stream(q.device)) == 0
    return o, lse


def _off(x, ref):
    ok = torch.isfinite(ref)
    assert torch.equal(torch.isfinite(x), ok)
    return ((x.double() - ref)[ok].norm() / ref[ok].norm()).item()


def _operands(H, L, d, contiguous):
    g = torch.Generator(device="cuda").manual_seed(L * d + H)
    q, k, v = (torch.empty(1, H, L, d, device="cuda").normal_(generator=g) for _ in range(3))
    kt = k.transpose(2, 3)
    return q, kt.contiguous() if contiguous else kt, v


@pytest.mark.parametrize("contiguous", [False, True])
@pytest.mark.parametrize("d", [32, 64, 128])
def test_no_further_off_than_fma_sums(d, contiguous):
    for mask, L, H in PATTERNS:
        acsr = ah.create_acsr(_mask(mask, L), 16, 0)
        q, kt, v = _operands(H, L, d, contiguous)
        for scale in (d ** -0.5, -1.0):
            ref_o, ref_lse = _exact(q, kt, v, acsr, scale)
            o, lse = _call(q, kt, v, acsr, scale)
            tile_o, tile_lse = _call(q, kt, v, acsr, scale, status=False)
            assert not torch.equal(o, tile_o), "the register tiles ran"
            assert _off(o, ref_o) <= _off(tile_o, ref_o), (L, H, scale)
            # both end in a value rounded to fp32 (2^-25 of it on average), of which the sums' errors are a part
            assert _off(lse, ref_lse) <= max(_off(tile_lse, ref_lse), 2 ** -24), (L, H, scale)


@pytest.mark.parametrize("d", [32, 64, 128])
def test_operands_on_16_bytes_give_the_same_bits(d):
    """Loads of 32 bytes where the operands allow them, of 16 elsewhere."""
    L, H = 520, 9
    acsr = ah.create_acsr(ah.create_windowed_mask(L, 70), 16, 0)
    for contiguous in (False, True):
        q, kt, v = _operands(H, L, d, contiguous)
        o, lse = _call(q, kt, v, acsr, 0.2)
        q4, k4, v4 = (torch.empty(t.numel() + 4, device="cuda")[4:].view(1, H, L, d).copy_(t) for t in (q, kt.transpose(2, 3), v))
        kt4 = k4.transpose(2, 3)
        if contiguous:
            kt4 = torch.empty(kt.numel() + 4, device="cuda")[4:].view(1, H, d, L).copy_(kt)
        o4, lse4 = _call(q4, kt4, v4, acsr, 0.2)
        assert torch.equal(o, o4) and torch.equal(lse, lse4)


def test_q_off_a_16_byte_boundary_stays_on_the_register_tiles():
    from test_gpu_tile_f32 import _Tiles
    L, H, d = 300, 40, 64
    acsr = ah.create_acsr(ah.create_windowed_mask(L, 40), 16, 0)
    q, kt, v = _operands(H, L, d, False)
    off = torch.empty(q.numel() + 1, device="cuda")[1:].view_as(q).copy_(q)
    tile_o, tile_lse = _call(q, kt, v, acsr, 0.125, status=False)
    o, lse = _call(off, kt, v, acsr, 0.125)
    s, tile_s = (torch.full((1, H, L, acsr[5]), float("nan"), device="cuda") for _ in range(2))
    n.sddmm(off, kt, s, *acsr[2:5], acsr[5])
    assert _Tiles(acsr, L, H, d).sddmm(q, kt, tile_s) == 0
    assert torch.equal(o, tile_o) and torch.equal(lse, tile_lse) and torch.equal(s, tile_s)


@pytest.mark.parametrize("op", ["fused", "sddmm", "spmm"])
def test_nothing_is_written_while_the_status_word_is_set(op):
    acsr = ah.create_acsr(ah.create_windowed_mask(300, 40), 16, 0)
    q, kt, v = _operands(40, 300, 64, False)
    meta, T = acsr[2:5], acsr[5]
    out = torch.full((1, 40, 300, T), 1e6, device="cuda") if op == "sddmm" else torch.full_like(q, 1e6)
    p = torch.rand(1, 40, 300, T, device="cuda")
    launch = {"fused": lambda: n.attention_fused(q, kt, v, out, *meta, 0.125), "sddmm": lambda: n.sddmm(q, kt, out, *meta, T),
              "spmm": lambda: n.spmm(p, v, out, *meta, T)}[op]
    n.classify(*meta)
    n.status_word(q.device).fill_(7)
    launch()
    torch.cuda.synchronize()
    assert (out == 1e6).all()
    with pytest.raises(RuntimeError):      # the launcher looks at the host copy of the word
        launch()
    launch()
    n.check_status_word(0)
    assert torch.isfinite(out).all() and not (out == 1e6).any()


def test_host_operands_while_the_status_word_is_set():
    """forward_host's results are never taken for good after a kernel gave up."""
    import r_attention
    H, L, d = 4, 300, 128
    attn = r_attention.RegularAttention(1, L, H, d, ah.create_windowed_mask(L, 40), 16, 16, 0, torch.float32, scale=d ** -0.5)
    q, k, v = (torch.randn(1, H, L, d).pin_memory() for _ in range(3))
    ref, out = torch.zeros(1, H, L, d).pin_memory(), torch.zeros(1, H, L, d).pin_memory()
    attn.forward_host(q, k, v, ref)
    torch.cuda.synchronize()
    n.status_word(attn.nnzs.device).fill_(7)
    attn.forward_host(q, k, v, out)        # a kernel that is started now passes the word on
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError):
        attn.forward_host(q, k, v, out)
    attn.forward_host(q, k, v, out)
    torch.cuda.synchronize()
    attn.check_status()
    assert torch.equal(out, ref) and ref.abs().sum() > 0


#        mask, L, heads: more than two waves of tiles of 32 rows
OPS = [
    (lambda L: ah.create_causal_windowed_mask(L, L - 1), 128, 75),
    (lambda L: ah.create_windowed_mask(L, 33), 129, 60),
    (lambda L: ah.create_windowed_mask(L, 100), 1004, 10),
    (lambda L: ah.create_windowed_mask(L, 40), 389, 23),
    (lambda L: ah.create_strided_mask(L, 8), 330, 19),                  # classes of 42 and 41 rows
    (lambda L: ah.create_dilated_mask(L, 40, 3), 301, 25),
    ("documents", 1000, 10),
]


def _slots(acsr, L, T):
    """Column of every slot (clamped) and whether it holds a non-zero."""
    lin, tr, nnz = (t.double() for t in acsr[2:5])
    stride, start = lin.round().clamp(min=1), (lin * tr).round()
    j = torch.arange(T, device="cuda").double()
    return (start[:, None] + j[None] * stride[:, None]).long().clamp(0, L - 1), j[None] < nnz[:, None]


@pytest.mark.parametrize("contiguous", [False, True])
@pytest.mark.parametrize("d", [32, 64, 128])
def test_sddmm_and_spmm(d, contiguous):
    from test_gpu_tile_f32 import _Tiles
    for mask, L, H in OPS:
        acsr = ah.create_acsr(_mask(mask, L), 16, 0)
        meta, T = acsr[2:5], acsr[5]
        cols, on = _slots(acsr, L, T)
        q, kt, v = _operands(H, L, d, contiguous)
        s = torch.full((1, H, L, T), float("nan"), device="cuda")
        n.sddmm(q, kt, s, *meta, T)
        n.check_status_word(0)
        tile, tile_s = _Tiles(acsr, L, H, d), torch.full_like(s, float("nan"))
        assert tile.sddmm(q, kt, tile_s) == 0 and not torch.equal(s, tile_s), "the register tiles ran"
        full = q.double() @ kt.double()
        ref = torch.gather(full, 3, cols[None, None].expand(1, H, L, T)) * on
        assert torch.count_nonzero(s * ~on) == 0, "padding slots must be zero"
        # what a chain of d fp32 additions, rounded to nearest, is off by on average: 0.5 sqrt(d / 3) 2^-24 of the result
        assert _off(s, ref) <= 0.5 * (d / 3) ** 0.5 * 2 ** -24, (L, H)
        # SpMM of probabilities; padding slots are not read
        p = torch.softmax(torch.where(on, ref * d ** -0.5, torch.tensor(float("-inf"), device="cuda").double()), -1)
        p = torch.where(on, torch.nan_to_num(p), torch.tensor(float("nan"), device="cuda").double()).float()
        o = torch.full((1, H, L, d), float("nan"), device="cuda")
        n.spmm(p, v, o, *meta, T)
        n.check_status_word(0)
        tile_o = torch.full_like(o, float("nan"))
        assert tile.spmm(p, v, tile_o) == 0 and not torch.equal(o, tile_o), "the register tiles ran"
        dense = torch.zeros(1, H, L, L, device="cuda", dtype=torch.double)
        dense.scatter_add_(3, cols[None, None].expand(1, H, L, T), torch.where(on, p, torch.zeros((), device="cuda")).double())
        # a rounded result is off by 2^-25 of itself on average, a few additions by as much
        assert _off(o, dense @ v.double()) <= 2 ** -23, (L, H)


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("window", [15, 63, 255])
def test_operands_of_one_sign(window, d):
    """Sums of positive numbers, where rounding towards zero does not average out."""
    from test_gpu_tile_f32 import _Tiles
    L, H = 1024, 10
    acsr = ah.create_acsr(ah.create_windowed_mask(L, window), 16, 0)
    meta, T = acsr[2:5], acsr[5]
    cols, on = _slots(acsr, L, T)
    tile = _Tiles(acsr, L, H, d)
    scale = d ** -0.5
    for form in ("uniform", "normal"):
        q, kt, v = (t.abs() if form == "normal" else torch.rand_like(t) for t in _operands(H, L, d, False))
        kt = kt.transpose(2, 3).contiguous().transpose(2, 3)
        nan = lambda *shape: torch.full(shape, float("nan"), device="cuda")
        s, tile_s, o = nan(1, H, L, T), nan(1, H, L, T), nan(1, H, L, d)
        n.sddmm(q, kt, s, *meta, T)
        assert tile.sddmm(q, kt, tile_s) == 0
        ref = torch.gather(q.double() @ kt.double(), 3, cols[None, None].expand(1, H, L, T)) * on
        assert _off(s, ref) <= _off(tile_s, ref), form
        # P V: each of the four additions of a step's 64 keys is short by half of 2^-23 of the sum so far on average, 2^-24 (1 + 3/4 + 1/2 + 1/4)
        # at most in all, and less the larger the mantissa; the steps are added with rounding
        p = torch.rand(1, H, L, T, device="cuda") * on
        n.spmm(p, v, o, *meta, T)
        dense = torch.zeros(1, H, L, L, device="cuda", dtype=torch.double).scatter_add_(3, cols[None, None].expand(1, H, L, T), p.double())
        assert _off(o, dense @ v.double()) <= 2 ** -23, form
        ref_o, ref_lse = _exact(q, kt, v, acsr, scale)
        o, lse = _call(q, kt, v, acsr, scale)
        assert _off(o, ref_o) <= 2 ** -23, form
        # a score is short by half of 2^-23 of itself, once; as much again for every other rounding together
        assert _off(lse, ref_lse) <= 1.5 * 2 ** -24, form


@pytest.mark.parametrize("power", [-140, -126, -118, 52, 100, 115])
def test_operands_of_any_magnitude(power):
    """All bits of a tiny operand count, down to fp32's denormal numbers, and one that is too large for its three pieces, or the sums of
    such, is not lost: relative errors are those of operands around 1, or of FMA sums where rows are computed again."""
    L, H, d = 129, 64, 64
    acsr = ah.create_acsr(ah.create_windowed_mask(L, 33), 16, 0)
    meta, T = acsr[2:5], acsr[5]
    cols, on = _slots(acsr, L, T)
    x, kt, v = _operands(H, L, d, False)
    up = 2.0 ** min(power, 100) * 2.0 ** max(power - 100, 0)
    big = x * up                           # (rounded to the denormals' spacing at 2^-140)
    other = kt * 2.0 ** (50 if power == 52 else 0)
    s = torch.full((1, H, L, T), float("nan"), device="cuda")
    n.sddmm(big, other, s, *meta, T)
    ref = torch.gather(big.double() @ other.double(), 3, cols[None, None].expand(1, H, L, T)) * on
    denormal = 2.0 ** -149 * ref.numel() ** 0.5 / ref.norm().item()        # what rounding the result to fp32 may add
    # a chain of d additions, each off by 2^-24 / sqrt(3) of a partial sum that grows with the root of their number
    assert _off(s, ref) <= (d / 6) ** 0.5 * 2 ** -24 + denormal
    p = torch.rand(1, H, L, T, device="cuda") * on
    dense = torch.zeros(1, H, L, L, device="cuda", dtype=torch.double)
    dense.scatter_add_(3, cols[None, None].expand(1, H, L, T), p.double())
    # sums of 67 products, at most 2^-25 of the largest partial sum each
    for pp, vv in ((p, v * up), (p * up, v)):
        o = torch.full((1, H, L, d), float("nan"), device="cuda")
        n.spmm(pp, vv, o, *meta, T)
        ref = (dense if pp is p else torch.zeros_like(dense).scatter_add_(3, cols[None, None].expand(1, H, L, T), pp.double())) @ vv.double()
        denormal = 2.0 ** -149 * 4 * ref.numel() ** 0.5 / ref.norm().item()      # ... at each of up to three steps
        assert _off(o, ref) <= 2 ** -22 + denormal
    # fused: V, and Q with a scale that makes up for it
    vv = v * up
    ref_o, ref_lse = _exact(x, kt, vv, acsr, 0.125)
    o, lse = _call(x, kt, vv, acsr, 0.125)
    denormal = 2.0 ** -149 * ref_o.numel() ** 0.5 / ref_o.norm().item()
    # scores as above, sums of 67 keys likewise, the exponentials' 2^-22 -- where rows are computed again with a chain of FMAs each
    bound = ((d / 6) ** 0.5 + (67 / 6) ** 0.5) * 2 ** -24 + 2 ** -22
    assert _off(o, ref_o) <= bound + denormal and _off(lse, ref_lse) <= 2 ** -22
    if -120 <= power <= 60:
        ref_o, ref_lse = _exact(big, kt, v, acsr, 0.125 / up)
        o, lse = _call(big, kt, v, acsr, 0.125 / up)
        assert _off(o, ref_o) <= bound and _off(lse, ref_lse) <= 2 ** -22
    n.check_status_word(0)


def test_tiny_scales_stay_on_the_register_tiles():
    acsr = ah.create_acsr(ah.create_windowed_mask(300, 40), 16, 0)
    q, kt, v = _operands(40, 300, 64, False)
    q, kt = q * 2.0 ** 35, kt * 2.0 ** 35
    for scale, same in ((2.0 ** -72, True), (0.0, True), (2.0 ** -60, False)):
        o, lse = _call(q, kt, v, acsr, scale)
        tile_o, tile_lse = _call(q, kt, v, acsr, scale, status=False)
        assert torch.equal(o, tile_o) == same and (not same or torch.equal(lse, tile_lse))


def test_sddmm_scores_that_are_not_finite():
    """An infinity is no sum of three bf16 numbers: such rows are computed again, as the row kernels give them."""
    L, H, d = 300, 40, 64
    acsr = ah.create_acsr(ah.create_windowed_mask(L, 20), 16, 0)
    meta, T = acsr[2:5], acsr[5]
    q, kt, _v = _operands(H, L, d, False)
    k = kt.transpose(2, 3)
    k[:, :, 50, 3], k[:, :, 120, 5], q[:, :, 200, 7] = float("inf"), float("nan"), float("-inf")
    q[:, :, 250, 0], k[:, :, 250, 0] = 3.4e38, 1e-30      # rounds to infinity in bf16
    s, rows = torch.empty(1, H, L, T, device="cuda"), torch.empty(1, H, L, T, device="cuda")
    n.sddmm(q, kt, s, *meta, T)
    n.sddmm(q, kt, rows, *meta, T, n.PATH_GENERIC)
    n.check_status_word(0)
    ok = torch.isfinite(rows)
    assert not ok.all() and torch.equal(torch.isfinite(s), ok)
    assert torch.equal(torch.isnan(s), torch.isnan(rows)) and torch.equal(s[torch.isinf(s)], rows[torch.isinf(rows)])
    assert (s[ok] - rows[ok]).abs().max() <= 1e-5 * rows[ok].abs().max()


FOREIGN_WORD = """
import torch
import acsr_helpers as ah
import splat_native as n
word = torch.full((1,), 7, dtype=torch.int32, device="cuda")
host = torch.zeros(1, dtype=torch.int32).pin_memory()
assert n._lib.splat_set_status_mirror(word.data_ptr(), host.data_ptr()) == 0
acsr = ah.create_acsr(ah.create_windowed_mask(300, 20), 16, 0)
q, k, v = (torch.randn(1, 40, 300, 64, device="cuda") for _ in range(3))
s, o = torch.full((1, 40, 300, acsr[5]), float("nan"), device="cuda"), torch.full_like(q, float("nan"))
for _ in range(2):        # (the first call takes the Python path)
    n.sddmm(q, k.transpose(2, 3), s.fill_(float("nan")), *acsr[2:5], acsr[5])
    n.spmm(s.nan_to_num(), v, o.fill_(float("nan")), *acsr[2:5], acsr[5])
    torch.cuda.synchronize()
    assert torch.isfinite(s).all() and torch.isfinite(o).all(), "not written"
assert word.item() == 7 and host.item() == 0, "another's word was used"
"""


def test_a_status_word_that_others_registered_is_not_used():
    env = dict(os.environ, PYTHONPATH=os.pathsep.join((SPLAT_DIR, ROOT)))
    done = subprocess.run([sys.executable, "-c", FOREIGN_WORD], env=env, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
