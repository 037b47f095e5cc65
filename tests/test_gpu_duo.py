"""GPU: the persistent two-tile kernel of d = 128, which takes over at 592 to 1776 tiles of 128 rows.  It multiplies and sums in the
order of the kernel with a tile per CTA, so the two agree bit for bit (and so do shards of a problem on either side of the
line); the first and last head are also compared with the CPU oracle."""
import pytest
import torch

from conftest import assert_close
from oracle import acsr_oracle as ao
from oracle import attention_oracle as at

pytestmark = pytest.mark.gpu

#        kind, L, p0, p1, batch * heads
PATTERNS = [
    (ao.PATTERN_CAUSAL_WINDOWED, 128, 40, 0, 740),     # one tile per head: neighbours never share keys; the fewest tiles
    (ao.PATTERN_CAUSAL_WINDOWED, 1000, 255, 0, 96),    # a short last tile
    (ao.PATTERN_CAUSAL_WINDOWED, 2048, 0, 0, 48),      # single-element rows only: nothing to multiply
    (ao.PATTERN_WINDOWED, 1536, 300, 0, 65),
    (ao.PATTERN_BLOCKED, 2048, 64, 0, 75),             # half steps at both ends
    (ao.PATTERN_STRIDED, 1024, 64, 0, 12),             # classes of 16 rows
    (ao.PATTERN_DILATED, 3072, 300, 2, 33),
]


# Left to the other kernel, too small or of too uneven tiles: forced.
FORCED = [
    (ao.PATTERN_CAUSAL_WINDOWED, 384, 200, 0, 397),    # odd number of tiles per head and in all: items across heads, half an item
    (ao.PATTERN_CAUSAL_WINDOWED, 2048, 1500, 0, 49),   # ranges that grow with the row
    (ao.PATTERN_BLOCKED, 2560, 777, 0, 40),            # neighbours whose ranges jump by more than the ring holds
    (ao.PATTERN_STRIDED, 4096, 4, 0, 37),              # triangular classes of eight tiles
    (ao.PATTERN_CAUSAL_WINDOWED, 128, 127, 0, 1),      # one tile
    (ao.PATTERN_CAUSAL_WINDOWED, 64, 9, 0, 1),         # half a tile
    (ao.PATTERN_CAUSAL_WINDOWED, 256, 255, 0, 1),      # two, an item each
    (ao.PATTERN_CAUSAL_WINDOWED, 120, 30, 0, 3),       # three, short
    (ao.PATTERN_CAUSAL_WINDOWED, 384, 0, 0, 1),        # nothing to multiply
    (ao.PATTERN_BLOCKED, 384, 128, 0, 1),
    (ao.PATTERN_STRIDED, 384, 3, 0, 1),                # three classes of one tile
    (ao.PATTERN_DILATED, 512, 100, 2, 1),
    (ao.PATTERN_WINDOWED, 128, 50, 0, 149),            # the fewest tiles that go in pairs, of two heads; the last item has one
    (ao.PATTERN_WINDOWED, 2048, 300, 0, 18),           # 288 tiles, 144 pairs: a wave, nothing to take over
    (ao.PATTERN_WINDOWED, 2048, 300, 0, 19),           # 304: 148 pairs and 8 single tiles that are taken over
]


def test_where_it_does_not_apply_it_refuses(monkeypatch):
    import acsr_helpers as ah
    import splat_native as n
    monkeypatch.setenv("SPLAT_B200_BAND_TILES", "4")
    for d, kind, L, p0, p1 in ((64, ao.PATTERN_CAUSAL_WINDOWED, 256, 31, 0), (128, ao.PATTERN_DILATED, 257, 30, 2)):
        acsr = ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0)
        q = torch.randn(1, 1, L, d, device="cuda").to(torch.bfloat16)
        out = torch.full_like(q, 5.0)
        with pytest.raises(RuntimeError):
            n.attention_fused(q, q.transpose(2, 3), q, out, acsr[2], acsr[3], acsr[4], 0.125, n.PATH_BAND)
        assert (out == 5.0).all()


@pytest.mark.parametrize("contiguous,dtype", [(False, torch.bfloat16), (True, torch.bfloat16), (False, torch.float16)])
@pytest.mark.parametrize("kind,L,p0,p1,H", PATTERNS + FORCED)
def test_duo_patterns(kind, L, p0, p1, H, contiguous, dtype, monkeypatch):
    import acsr_helpers as ah
    import splat_native as n
    if contiguous and kind in (ao.PATTERN_STRIDED, ao.PATTERN_DILATED):
        pytest.skip("a contiguous K^T of a strided pattern is copied to rows first")
    d, scale = 128, 128 ** -0.5
    g = torch.Generator(device="cuda").manual_seed(L + p0)
    acsr = ah.create_acsr(ah.PatternMask(kind, L, p0, p1), 16, 0)
    q, k, v = (torch.randn(1, H, L, d, device="cuda", generator=g).to(dtype) for _ in range(3))
    kt = k.transpose(2, 3)
    kt = kt.contiguous() if contiguous else kt

    def run(lse):
        out = torch.full((1, H, L, d), float("nan"), dtype=dtype, device="cuda")
        n.attention_fused(q, kt, v, out, acsr[2], acsr[3], acsr[4], scale, n.PATH_BAND, lse=lse)
        n.check_status_word(0)
        return out

    if (kind, L, p0, p1, H) in FORCED:
        monkeypatch.setenv("SPLAT_B200_BAND_TILES", "4")
    else:
        monkeypatch.delenv("SPLAT_B200_BAND_TILES", raising=False)
        plan = n.classify(acsr[2], acsr[3], acsr[4])
        assert n.band_table(acsr[2], acsr[3], acsr[4], L) is not None
        assert n.band_kernel_choice(H, L, d, plan) == 4, "this kernel is not the one that runs"
    lse, lse_one = (torch.full((1, H, L), float("nan"), device="cuda") for _ in range(2))
    out, plain = run(lse), run(None)
    monkeypatch.setenv("SPLAT_B200_BAND_TILES", "1")
    one = run(lse_one)
    assert torch.equal(out, plain), "the log-sum-exp output changes the result"
    assert torch.equal(out, one)
    assert torch.equal(lse, lse_one)
    meta = ao.metadata_from_pattern(kind, L, p0, p1, 16)
    ends = sorted({0, H - 1})
    qc, kc, vc = (t[:, ends].cpu() for t in (q, k, v))
    assert_close(out[:, ends], at.attention_acsr(qc, kc.transpose(2, 3), vc, meta, meta["trailing_dim"], scale), dtype)


def test_duo_unscaled_scores_need_the_running_max(monkeypatch):
    """scale = 1 gives scores of sigma ~ 11: the rescale of O, also while the other tile is in mid-step."""
    import acsr_helpers as ah
    import splat_native as n
    B, H, L, d = 1, 48, 2048, 128
    acsr = ah.create_acsr(ah.create_causal_windowed_mask(L, 511), 16, 0)
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(B, H, L, d, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    outs = []
    for variant in (None, "1"):
        if variant:
            monkeypatch.setenv("SPLAT_B200_BAND_TILES", variant)
        else:
            monkeypatch.delenv("SPLAT_B200_BAND_TILES", raising=False)
            assert n.band_kernel_choice(B * H, L, d, n.classify(acsr[2], acsr[3], acsr[4])) == 4
        outs.append(torch.full_like(q, float("nan")))
        n.attention_fused(q, k.transpose(2, 3), v, outs[-1], acsr[2], acsr[3], acsr[4], 1.0, n.PATH_BAND)
        n.check_status_word(0)
    assert torch.isfinite(outs[0].float()).all() and torch.equal(*outs)


@pytest.mark.parametrize("contiguous", [False, True])
def test_duo_single_rows_do_not_hold_up_the_log_sum_exp(contiguous, monkeypatch):
    """One row with one key per head, whose score is formed apart: a fraction of the call, not a multiple (5 at worst once)."""
    import acsr_helpers as ah
    import splat_native as n
    H, L, d = 320, 512, 128
    acsr = ah.create_acsr(ah.create_causal_windowed_mask(L, 127), 16, 0)
    q = torch.randn(1, H, L, d, device="cuda").to(torch.bfloat16)
    kt = q.transpose(2, 3).contiguous() if contiguous else q.transpose(2, 3)
    out, lse = torch.empty_like(q), torch.empty(1, H, L, device="cuda")
    monkeypatch.setenv("SPLAT_B200_BAND_TILES", "4")

    def seconds(extra):
        best = float("inf")
        for _ in range(20):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda._sleep(200_000)          # (the calls are in the queue before the first begins)
            e[0].record()
            for _ in range(4):
                n.attention_fused(q, kt, q, out, acsr[2], acsr[3], acsr[4], d ** -0.5, n.PATH_BAND, lse=extra)
            e[1].record()
            e[1].synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best

    assert seconds(lse) < 1.6 * seconds(None)
