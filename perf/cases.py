"""What a user of this package has it do, as measurable cases.

Five kinds of call, all through the modules of the SPLAT directory:

  fused      RegularAttention.forward, one kernel per call (the default of the module)
  module     RegularAttention.forward with fused=False: SDDMM, softmax and SpMM with the score and
             probability arrays kept in the module's buffers
  launchers  rsddmm_launcher, rsoftmax_launcher, rspmm_launcher called one by one, as a program
             written against the reference's functions does
  host       RegularAttention.forward_host: pinned host operands and result
  metadata   create_acsr of an explicit mask on the GPU

A case gives the kind, the data type, (B, H, L, d), the sparsity pattern with its parameters, how K^T
is handed over ("view": the transposed view of a (B, H, L, d) tensor, "contiguous": the
reference's own (B, H, d, L) array) and whether the log-sum-exp output is asked for.
"""
import math
import os
import sys

import numpy as np
import torch

_SPLAT = os.path.join(os.getcwd(), "triton-fun_b200", "SPLAT")
if _SPLAT not in sys.path:
    sys.path.insert(0, _SPLAT)

import acsr_helpers as ah  # noqa: E402
from r_attention import RegularAttention  # noqa: E402
from r_sddmm import rsddmm_launcher, rsddmm_preamble  # noqa: E402
from r_softmax import rsoftmax_launcher, rsoftmax_preamble  # noqa: E402
from r_spmm import rspmm_launcher, rspmm_preamble  # noqa: E402

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
BLOCK = 16                     # BLOCK_SIZE_Y = BLOCK_SIZE_X of the benchmark and the tests


def _attn(name, kind, dtype, B, H, L, d, pattern, p0, p1=0, kt="view", lse=False, spread=1.0):
    return {"name": name, "kind": kind, "dtype": dtype, "B": B, "H": H, "L": L, "d": d, "pattern": pattern,
            "p0": p0, "p1": p1, "kt": kt, "lse": lse, "spread": spread}


def listed():
    return [
        # Smallest configuration of the benchmark: a call whose latency is all that counts.
        _attn("fused_fp32_tiny", "fused", "fp32", 1, 2, 256, 32, "causal_windowed", 31),
        # A short prompt through one layer: a few tiles, latency and launch bound.
        _attn("fused_bf16_short", "fused", "bf16", 1, 8, 512, 64, "causal_windowed", 127),
        # Local causal attention of a training batch (configuration 2 of the benchmark).
        _attn("fused_fp16_local", "fused", "fp16", 4, 16, 4096, 64, "causal_windowed", 255),
        # Column-strided attention (configuration 3): little arithmetic, all bandwidth.
        _attn("fused_bf16_strided", "fused", "bf16", 2, 32, 8192, 128, "strided", 64),
        # Dilated window (configuration 4): bandwidth and arithmetic in balance.
        _attn("fused_bf16_dilated", "fused", "bf16", 1, 32, 16384, 128, "dilated", 512, 2, spread=0.5),
        # Long-context prefill (configuration 5, the benchmark's headline): the largest call.
        _attn("fused_bf16_long", "fused", "bf16", 8, 64, 32768, 128, "causal_windowed", 1023),
        # Bidirectional window over a batch padded to an odd length, the reference's K^T layout, with the
        # log-sum-exp a later merge or backward pass starts from.
        _attn("fused_bf16_ragged_lse", "fused", "bf16", 3, 12, 3000, 128, "windowed", 200, kt="contiguous",
              lse=True),
        # The reference's own data type and layout at an ordinary size.
        _attn("fused_fp32_local", "fused", "fp32", 2, 16, 4096, 64, "causal_windowed", 255, kt="contiguous"),
        # Three-kernel forward at the size of configuration 2: scores and probabilities are wanted too.
        _attn("module_fp16_local", "module", "fp16", 4, 16, 4096, 64, "causal_windowed", 255),
        # The reference's comparison sweep (L = 1024, windowed) through its own launchers, fp32.
        _attn("launchers_fp32_sweep", "launchers", "fp32", 1, 8, 1024, 64, "windowed", 64, kt="contiguous"),
        # Operands that live on the host: one chunk of heads in, attention, result out.
        _attn("host_bf16", "host", "bf16", 2, 16, 8192, 128, "causal_windowed", 511),
        # Metadata of a user's explicit mask (ragged windows, e.g. document boundaries).
        {"name": "metadata_mask", "kind": "metadata", "L": 8192, "width": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["fused", "module", "launchers", "host", "metadata"], [55, 12, 12, 8, 13])[0]
    if kind == "metadata":
        L = _log(rng, 128, 16384)
        return {"kind": kind, "L": L, "width": _log(rng, 8, max(9, L // 4))}
    dtype = rng.choices(["fp32", "fp16", "bf16"], [25, 30, 45])[0]
    L = _log(rng, 128, 32768)
    if rng.random() < 0.5:
        L = max(128, L // 128 * 128)
    d = rng.choices([32, 64, 128], [15, 40, 45])[0]
    pattern = rng.choices(["causal_windowed", "windowed", "blocked", "strided", "dilated"], [35, 20, 15, 15, 15])[0]
    p1 = 0
    if pattern == "strided":
        p0 = _log(rng, 4, 128)
    elif pattern == "dilated":
        p0, p1 = _log(rng, 16, 1024), rng.choice([2, 3, 4, 8])
    else:
        p0 = _log(rng, 16, max(17, min(L // 2, 1536)))
        if pattern == "causal_windowed" and rng.random() < 0.7:
            p0 = max(15, (p0 + 1) // 16 * 16 - 1)      # window width a round number
    case = _attn("", kind, dtype, 1, 1, L, d, pattern, p0, p1,
                 kt="view" if kind == "host" or rng.random() < 0.6 else "contiguous",
                 lse=kind == "fused" and rng.random() < 0.2,
                 spread=rng.choice([0.5, 1.0]))
    del case["name"]
    # As many heads as a batch brings along, within what the kind of call is used for.
    most = 3e10 if dtype == "fp32" else (1e12 if kind == "fused" and pattern.endswith("windowed") else 2e11)
    bytes_most = 4e8 if kind == "host" else 4e9
    heads = _log(rng, 1, 256)
    one = work(case)
    heads = max(1, min(heads, int(most / one["flops"]), int(bytes_most / one["bytes"])))
    case["B"] = rng.choice([b for b in (1, 2, 3, 4) if b <= heads])
    case["H"] = max(1, heads // case["B"])
    return case


def _counts(case):
    """Non-zeros of every row of the pattern."""
    L, p0, p1 = case["L"], case["p0"], case["p1"]
    i = np.arange(L, dtype=np.int64)
    if case["pattern"] == "causal_windowed":
        return np.minimum(i, p0) + 1
    if case["pattern"] == "windowed":
        return np.minimum(i + p0 + 1, L) - np.maximum(i - p0, 0)
    if case["pattern"] == "blocked":
        start = np.where(i < p0, 0, (i // p0 - 1) * p0)
        return np.minimum(np.where(i < p0, p0, start + 2 * p0), L) - start
    if case["pattern"] == "strided":
        return i // p0 + 1
    return np.minimum(p0, i // p1 + 1)


def _mask(case):
    L, p0, p1 = case["L"], case["p0"], case["p1"]
    if case["pattern"] == "dilated":
        return ah.create_dilated_mask(L, p0, p1)
    return {"causal_windowed": ah.create_causal_windowed_mask, "windowed": ah.create_windowed_mask,
            "blocked": ah.create_blocked_mask, "strided": ah.create_strided_mask}[case["pattern"]](L, p0)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "metadata":
        L = case["L"]
        row = torch.arange(L, device="cuda")
        back = torch.randint(0, case["width"], (L,), device="cuda", generator=g)
        ahead = torch.randint(0, case["width"], (L,), device="cuda", generator=g)
        lo, hi = (row - back)[:, None], (row + ahead)[:, None]
        return {"kind": "metadata", "mask": ((row[None] >= lo) & (row[None] <= hi)).to(torch.uint8)}
    B, H, L, d = case["B"], case["H"], case["L"], case["d"]
    dtype = DTYPES[case["dtype"]]
    # normal values as a projection gives them; configuration 4 of the benchmark has them at half the spread
    q, k, v = (torch.empty(B, H, L, d, dtype=dtype, device="cuda").normal_(0.0, case["spread"], generator=g)
               for _ in range(3))
    mask, scale = _mask(case), d ** -0.5
    state = {"kind": case["kind"]}
    if case["kind"] == "host":
        state["attn"] = RegularAttention(B, L, H, d, mask, BLOCK, BLOCK, 0, dtype, scale=scale)
        state["io"] = [t.cpu().pin_memory() for t in (q, k, v)] + [torch.empty(B, H, L, d, dtype=dtype).pin_memory()]
        return state
    kt = k.transpose(2, 3)
    if case["kt"] == "contiguous":
        kt = kt.contiguous()
    if case["kind"] == "launchers":
        acsr = ah.create_acsr(mask, BLOCK, 0)
        scores = (B, H, L, acsr[5])
        state.update(q=q, kt=kt, v=v, acsr=acsr, scale=scale,
                     sddmm=rsddmm_preamble(mask, scores, BLOCK, BLOCK, 0, dtype),
                     softmax=rsoftmax_preamble(mask, scores, BLOCK, 0, dtype),
                     spmm=rspmm_preamble(mask, (B, H, L, d), BLOCK, BLOCK, 0, dtype))
        return state
    state["attn"] = RegularAttention(B, L, H, d, mask, BLOCK, BLOCK, 0, dtype, scale=scale,
                                     fused=case["kind"] == "fused", lse=case["lse"])
    state["x"] = [q, kt, v]
    return state


def run(state):
    kind = state["kind"]
    if kind == "fused":
        attn = state["attn"]
        o = attn(state["x"])
        return o if attn.lse is None else (o, attn.lse)
    if kind == "module":
        attn = state["attn"]
        o = attn(state["x"])
        return attn.rsddmm_output, attn.rsoftmax_output, o
    if kind == "metadata":
        return ah.create_acsr(state["mask"], BLOCK, 0)
    if kind == "host":
        q, k, v, o = state["io"]
        out = state["attn"].forward_host(q, k, v, o)
        torch.cuda.current_stream().synchronize()      # as the method asks for before the result is read
        return out
    d2s_lin, d2s_tr, s2d_lin, s2d_tr, nnzs, trailing, span0, span1 = state["acsr"]
    s, s_grid, tb_x, tb_y = state["sddmm"]
    rsddmm_launcher(state["q"], state["kt"], s, d2s_lin, d2s_tr, s2d_lin, s2d_tr, trailing, nnzs, s_grid, tb_x,
                    tb_y, BLOCK, BLOCK)
    p_grid, p, _, pow_two = state["softmax"]
    rsoftmax_launcher(s, p, d2s_lin, d2s_tr, s2d_lin, s2d_tr, trailing, pow_two, nnzs, p_grid, BLOCK,
                      scale=state["scale"])
    o, o_grid, _ = state["spmm"]
    rspmm_launcher(p, state["v"], o, d2s_lin, d2s_tr, s2d_lin, s2d_tr, span0, span1, trailing, nnzs, o_grid, BLOCK,
                   BLOCK)
    return s, p, o


def work(case):
    if case["kind"] == "metadata":      # the mask read once; five vectors and two per 16 rows written
        L = case["L"]
        return {"bytes": L * L + 20 * L + 8 * -(-L // BLOCK), "flops": 0}
    bh, L, d = case["B"] * case["H"], case["L"], case["d"]
    e = 4 if case["dtype"] == "fp32" else 2
    nnz = _counts(case)
    nbytes = 4 * bh * L * d * e         # Q, K, V read, O written
    if case["lse"]:
        nbytes += 4 * bh * L
    if case["kind"] in ("module", "launchers"):
        nbytes += 2 * bh * L * int(nnz.max()) * e      # scores and probabilities written
    return {"bytes": nbytes, "flops": 4 * bh * int(nnz.sum()) * d}


def tolerance(case):
    if case["kind"] == "metadata":
        return "exact"
    # 32-bit sums in any order; 16-bit results and probabilities rounded once (2^-11, 2^-8)
    return {"rel": {"fp32": 1e-5, "fp16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
