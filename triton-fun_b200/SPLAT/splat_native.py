"""ctypes binding of libsplat_b200.so (the C ABI declared in include/splat_b200.h).

There is no fallback: if the library is missing this module raises at import, and every wrapper
turns a non-zero status into ``RuntimeError``.  Build the library with
``python triton-fun_b200/build.py`` (nvcc, sm_100a).
"""
from __future__ import annotations

import contextlib
import ctypes
import os
import threading

import torch

_PKG_DIR = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB_PATH = os.environ.get("SPLAT_B200_LIB") or os.path.join(_PKG_DIR, "libsplat_b200.so")

if not os.path.exists(LIB_PATH):
    raise ImportError(
        f"{LIB_PATH} not found: build it with `python {os.path.join(_PKG_DIR, 'build.py')}` "
        "(this package has no CPU or eager fallback)")

_lib = ctypes.CDLL(LIB_PATH)
try:
    import splat_host as _host      # native host path of the launchers (csrc/host_binding.cpp)
except ImportError as e:
    raise ImportError(f"the splat_host extension is missing or does not load ({e}): build it with "
                      f"`python {os.path.join(_PKG_DIR, 'build.py')}`") from e

_i32, _i64, _f32, _vp = ctypes.c_int32, ctypes.c_int64, ctypes.c_float, ctypes.c_void_p

# name -> argtypes; every function returns int32 except splat_status_string
SIGNATURES = {
    "splat_version": [],
    "splat_mask_row_summary_u8": [_vp, _i64, _i64, _i64, _vp, _vp],
    "splat_pattern_row_summary": [_i32, _i64, _i64, _i64, _vp, _vp],
    "splat_pattern_mask_u8": [_i32, _i64, _i64, _i64, _vp, _i64, _vp],
    "splat_acsr_from_row_summary": [_vp, _i64, _i64, _i32] + [_vp] * 8 + [_vp],
    "splat_acsr_classify": [_vp, _vp, _vp, _i64, _vp, _vp],
    "splat_sddmm": [_vp, _vp, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _i64,
                    _i32, _vp],
    "splat_softmax": [_vp, _vp, _vp, _i64, _i64, _i64, _f32, _i32, _vp],
    "splat_spmm": [_vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _i64, _i32, _vp],
    "splat_attention_fused": [_vp, _vp, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _vp, _i64, _i64,
                              _i64, _i64, _f32, _i32, _i32, _vp, _vp, _vp],
    "splat_attention_fused_ex": [_vp, _vp, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _vp, _i64, _i64,
                                 _i64, _i64, _f32, _i32, _i32, _vp, _vp, _vp, _vp],
    "splat_attention_fused_lse": [_vp, _vp, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64,
                                  _i64, _i64, _f32, _i32, _i32, _vp, _vp, _vp, _vp],
    "splat_sddmm_band": [_vp, _vp, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _i64,
                         _i32, _vp, _vp, _vp],
    "splat_spmm_band": [_vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _i64, _i32, _vp, _vp,
                        _vp],
    "splat_sddmm_tile": [_vp, _vp, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _i64,
                         _i32, _vp, _vp],
    "splat_spmm_tile": [_vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _i64, _i32, _vp, _vp],
    "splat_sddmm_tile_status": [_vp, _vp, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _i64,
                                _i32, _vp, _vp, _vp],
    "splat_spmm_tile_status": [_vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _i64, _i32, _vp, _vp, _vp],
    "splat_sddmm_band_table": [_vp, _vp, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _i64,
                               _i32, _vp, _vp, _vp, _vp],
    "splat_spmm_band_table": [_vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _i64, _i32, _vp, _vp,
                              _vp, _vp],
    "splat_selftest_bounded_wait": [_vp, _i64, _vp],
    "splat_debug_check_indices": [_vp],
    "splat_set_status_mirror": [_vp, _vp],
    "splat_acsr_from_mask_u8": [_vp, _i64, _i64, _i64, _i32] + [_vp] * 9 + [_vp],
    "splat_transpose_16": [_vp, _vp, _i64, _i64, _i64, _vp],
    "splat_attention_host": [_vp] * 5 + [_i64] + [_vp] * 3 + [_i64] * 3 + [_f32, _i32, _i32] + [_vp] * 8,
    "splat_band_kernel_choice": [_i64, _i64, _i64, _vp, _i32],
    "splat_band_table": [_vp, _vp, _vp, _i64, _i64, _vp, _vp],
    "splat_attention_fused_table": [_vp, _vp, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64,
                                    _i64, _i64, _f32, _i32, _i32, _vp, _vp, _vp, _vp, _vp],
    "splat_attention_noalloc": [_vp, _vp, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _vp, _i64, _i64,
                                _i64, _i64, _i64, _f32, _i32, _vp],
}
for _name, _args in SIGNATURES.items():
    _fn = getattr(_lib, _name)
    _fn.argtypes = _args
    _fn.restype = _i32
_lib.splat_status_string.argtypes = [_i32]
_lib.splat_status_string.restype = ctypes.c_char_p

PATTERN_BLOCKED, PATTERN_WINDOWED, PATTERN_CAUSAL_WINDOWED, PATTERN_STRIDED, PATTERN_DILATED = range(5)
PATH_AUTO, PATH_GENERIC, PATH_BAND = 0, 1, 2
NOALLOC_SCRATCH_BYTES = 64 << 20     # SPLAT_NOALLOC_SCRATCH_BYTES in include/splat_b200.h
DTYPES = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}


def status_string(code: int) -> str:
    return _lib.splat_status_string(int(code)).decode()


def check(code: int, what: str) -> None:
    if code != 0:
        raise RuntimeError(f"{what}: splat status {code} ({status_string(code)})")


def version() -> int:
    return _lib.splat_version()


def resolve_device(gpu_id) -> torch.device:
    """GPU_ID of the reference API: an int or a torch/cuda device.  'cpu' is rejected."""
    dev = torch.device("cuda", gpu_id) if isinstance(gpu_id, int) else torch.device(gpu_id)
    if dev.type != "cuda":
        raise ValueError(f"device {gpu_id!r}: this implementation runs on CUDA devices only "
                         "(there is no CPU path)")
    if dev.index is None:
        dev = torch.device("cuda", torch.cuda.current_device())
    return dev


def _stream(dev: torch.device) -> int:
    return torch.cuda.current_stream(dev).cuda_stream


def dtype_code(dt: torch.dtype) -> int:
    try:
        return DTYPES[dt]
    except KeyError:
        raise TypeError(f"unsupported dtype {dt}; expected float32, float16 or bfloat16") from None


def _f32_vec(t: torch.Tensor, n: int, name: str) -> int:
    if t.dtype != torch.float32 or not t.is_cuda or not t.is_contiguous() or t.numel() < n:
        raise ValueError(f"{name} must be a contiguous float32 CUDA tensor of at least {n} elements")
    return t.data_ptr()


# ----------------------------------------------------------------------------------------------
# metadata
# ----------------------------------------------------------------------------------------------
def mask_row_summary(mask_u8: torch.Tensor) -> torch.Tensor:
    """(rows, cols) uint8 CUDA mask -> int32 (4, rows): first, second, last set column, count."""
    assert mask_u8.is_cuda and mask_u8.dtype == torch.uint8 and mask_u8.dim() == 2
    if mask_u8.stride(1) != 1:
        mask_u8 = mask_u8.contiguous()
    rows, cols = mask_u8.shape
    out = torch.empty((4, rows), dtype=torch.int32, device=mask_u8.device)
    with torch.cuda.device(mask_u8.device):
        check(_lib.splat_mask_row_summary_u8(mask_u8.data_ptr(), rows, cols, mask_u8.stride(0),
                                             out.data_ptr(), _stream(mask_u8.device)),
              "splat_mask_row_summary_u8")
    return out


def pattern_row_summary(kind: int, n: int, p0: int, p1: int, dev: torch.device) -> torch.Tensor:
    out = torch.empty((4, n), dtype=torch.int32, device=dev)
    with _on(dev):
        check(_lib.splat_pattern_row_summary(kind, n, p0, p1, out.data_ptr(), _stream(dev)),
              "splat_pattern_row_summary")
    return out


def pattern_mask(kind: int, n: int, p0: int, p1: int, dev: torch.device) -> torch.Tensor:
    out = torch.empty((n, n), dtype=torch.uint8, device=dev)
    with _on(dev):
        check(_lib.splat_pattern_mask_u8(kind, n, p0, p1, out.data_ptr(), out.stride(0) if n else 0,
                                         _stream(dev)), "splat_pattern_mask_u8")
    return out


def acsr_from_row_summary(rows_i32: torch.Tensor, n_cols: int, block_height: int):
    """-> (dTos_lin, dTos_tr, sTod_lin, sTod_tr, nnzs, trailing_dim, span_start, span_end)."""
    dev = rows_i32.device
    n_rows = rows_i32.shape[1]
    n_blocks = -(-n_rows // block_height)
    vec = [torch.empty(n_rows, dtype=torch.float32, device=dev) for _ in range(5)]
    spans = [torch.empty(n_blocks, dtype=torch.float32, device=dev) for _ in range(2)]
    td = torch.empty(1, dtype=torch.int32, device=dev)
    with _on(dev):
        check(_lib.splat_acsr_from_row_summary(
            rows_i32.data_ptr(), n_rows, n_cols, block_height, *[v.data_ptr() for v in vec],
            spans[0].data_ptr(), spans[1].data_ptr(), td.data_ptr(), _stream(dev)),
            "splat_acsr_from_row_summary")
    return (*vec, int(td.item()), spans[0], spans[1])


_SET_UP = threading.Lock()      # what a device gets once: kernels and the native path keep the addresses
_MASK_SLOTS = 16
_MASK_WORK: dict = {}


def acsr_from_mask(mask_u8: torch.Tensor, block_height: int):
    """acsr_from_row_summary(mask_row_summary(mask)) in one kernel, or None where that does not apply (block
    heights outside 4 .. 64, no unit column stride, another current device)."""
    dev = mask_u8.device
    if dev.index not in _MASK_WORK:
        with _SET_UP:
            if dev.index not in _MASK_WORK:        # scratch of the calls in progress: 16 slots, device and page-locked host
                with torch.cuda.device(dev):
                    work = torch.zeros(2 * _MASK_SLOTS, dtype=torch.int32, device=dev)
                    torch.cuda.current_stream(dev).synchronize()
                    host = torch.zeros(_MASK_SLOTS, dtype=torch.int32).pin_memory()
                _host.set_mask_work(dev.index, _MASK_SLOTS, work.data_ptr(), host.data_ptr())
                _MASK_WORK[dev.index] = (work, host)
    return _host.acsr_from_mask(mask_u8, block_height)


def attention_host(q, k, v, out, stage: dict, sTod_lin, sTod_tr, nnzs, scale: float, path: int, plan) -> None:
    """Host tensors (B,H,L,d) through the device in chunks; stage as RegularAttention.forward_host keeps it."""
    dev = nnzs.device
    B, H, L, d = q.shape
    if _may_give_up(q, path):
        _raise_if_gave_up(dev)
    sw = status_word(dev)
    table = band_table(sTod_lin, sTod_tr, nnzs, L) if _band_candidate(q, path) else None
    ran = ctypes.c_int32(0)
    plan_arr = (ctypes.c_int32 * 8)(*plan)
    _debug_before(dev)
    with _on(dev):
        rc = _lib.splat_attention_host(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), stage["staging"], stage["chunk"],
            _f32_vec(sTod_lin, L, "sTod_lin"), _f32_vec(sTod_tr, L, "sTod_tr"), _f32_vec(nnzs, L, "nnzs"), B * H, L, d,
            float(scale), dtype_code(q.dtype), int(path), ctypes.cast(plan_arr, _vp) if path != PATH_GENERIC else None,
            table, sw.data_ptr(), ctypes.byref(ran), stage["s_in"].cuda_stream, _stream(dev),
            stage["s_out"].cuda_stream, stage["events"])
        # the caller may drop its tensors now: their page-locked blocks are reused only when the copies are done
        for t in (q, k, v):
            _host.record_pinned(t, *stage["s_in_key"])
        _host.record_pinned(out, *stage["s_out_key"])
    check(rc, "splat_attention_host")
    if ran.value != PATH_BAND and q.dtype != torch.float32 and q.numel() > 0 and path == PATH_AUTO:
        _warn_cuda_core_16bit("attention")
    if os.environ.get("SPLAT_B200_DEBUG"):
        check_status_word(dev)


def _plan_key(sTod_lin, sTod_tr, nnzs) -> tuple:
    return (id(sTod_lin), id(sTod_tr), sTod_lin._version, sTod_tr._version, nnzs._version, nnzs.numel())


def _known_plan(sTod_lin, sTod_tr, nnzs):
    """What classify() remembers of these metadata, or None if it has not seen them as they are."""
    hit = getattr(nnzs, "_splat_plan", None)
    return hit if hit is not None and hit[0] == _plan_key(sTod_lin, sTod_tr, nnzs) else None


def classify(sTod_lin: torch.Tensor, sTod_tr: torch.Tensor, nnzs: torch.Tensor) -> tuple:
    """Host copy of the 8 plan ints of ``splat_acsr_classify``.  The result is remembered ON the ``nnzs`` tensor
    object (with the identities and versions of all three tensors), so it lives exactly as long as that
    metadata and is recomputed if any of them is modified in place."""
    hit = _known_plan(sTod_lin, sTod_tr, nnzs)
    if hit is not None:
        return hit[1]
    key = _plan_key(sTod_lin, sTod_tr, nnzs)
    dev = nnzs.device
    status_word(dev)        # (the launches that follow may be captured, and setting it up synchronises)
    n = nnzs.numel()
    plan = torch.empty(8, dtype=torch.int32, device=dev)
    with _on(dev):
        check(_lib.splat_acsr_classify(_f32_vec(sTod_lin, n, "sTod_lin"), _f32_vec(sTod_tr, n, "sTod_tr"),
                                       _f32_vec(nnzs, n, "nnzs"), n, plan.data_ptr(), _stream(dev)),
              "splat_acsr_classify")
    host = tuple(int(v) for v in plan.cpu().tolist())
    # keep the two companions alive with the cache entry so their ids cannot be reused
    nnzs._splat_plan = (key, host, sTod_lin, sTod_tr, None, 0)
    return host


def band_table(sTod_lin, sTod_tr, nnzs, n_rows: int):
    """Address of the band table (``splat_band_table``) of classified metadata, which lives with their plan; made by
    the first call that reads it.  None if the pattern has none, if the
    metadata have changed since classify() or have more rows than the operands -- or for a captured launch,
    which has to work with the metadata as they are at the replay."""
    hit = _known_plan(sTod_lin, sTod_tr, nnzs)
    dev = nnzs.device
    if hit is None or hit[4] is False or nnzs.numel() != n_rows:
        return None
    stream = torch.cuda.current_stream(dev)
    if stream.cuda_stream != 0 and _capturing(dev):        # (the legacy stream is never captured)
        return None
    if hit[4] is None:
        plan, n = hit[1], n_rows
        stride = plan[1] if plan[7] > 0 else 1
        if not (0 < n <= 2**31 - 1 and (plan[7] == 0 or plan[1] == plan[2]) and plan[3] == 0 and plan[5] <= n and stride <= 65535):
            nnzs._splat_plan = hit[:4] + (False, 0)
            return None
        tiles = -(-(-(-n // stride)) // 128) * stride
        table = torch.empty(2 * (n + tiles), dtype=torch.int32, device=dev)
        with _on(dev):
            check(_lib.splat_band_table(sTod_lin.data_ptr(), sTod_tr.data_ptr(), nnzs.data_ptr(), n, stride,
                                        table.data_ptr(), stream.cuda_stream), "splat_band_table")
            # any stream may use it.  (An event for the others to wait for instead: 30 us where metadata are kept, for its creation)
            stream.synchronize()
        hit = nnzs._splat_plan = hit[:4] + (table, stream.cuda_stream)
    if hit[5] != stream.cuda_stream:      # the table is nobody's tensor but ours: its use elsewhere is ours to record
        hit[4].record_stream(stream)
    return hit[4].data_ptr()


def band_kernel_choice(bh: int, n_rows: int, d: int, plan, has_band_table: bool = True) -> int:
    """``splat_band_kernel_choice`` for a plan of classify(): the fused kernel that a band problem gets."""
    return _lib.splat_band_kernel_choice(bh, n_rows, d, ctypes.cast((ctypes.c_int32 * 8)(*plan), _vp), int(has_band_table))


_STATUS_WORDS: dict = {}
_STATUS_MIRRORS: dict = {}


def status_word(dev: torch.device) -> torch.Tensor:
    """Per-device int32 the tensor-core kernels set when one of their bounded waits gives up.  Beside it
    lives a pinned host copy that a kernel started while the word is set writes itself, so that the host
    can look at it without synchronising or copying anything on the normal path."""
    key = (dev.type, dev.index)
    t = _STATUS_WORDS.get(key)
    if t is not None:
        return t
    with _SET_UP:
        t = _STATUS_WORDS.get(key)
        if t is not None:
            return t
        with torch.cuda.device(dev):
            t = torch.zeros(1, dtype=torch.int32, device=dev)
            torch.cuda.current_stream(dev).synchronize()
            host = torch.zeros(1, dtype=torch.int32).pin_memory()
            check(_lib.splat_set_status_mirror(t.data_ptr(), host.data_ptr()), "splat_set_status_mirror")
        _STATUS_MIRRORS[key] = {"host": host, "value": ctypes.c_int32.from_address(host.data_ptr())}
        _STATUS_WORDS[key] = t
        _host.set_status(dev.index, t.data_ptr(), host.data_ptr())
    return t


def _raise_if_gave_up(dev: torch.device) -> None:
    """Start of every tensor-core launcher: if an earlier launch on this device reported a
    timed-out wait (the kernels do nothing while the word is set), clear the word and raise
    instead of silently returning stale outputs.  Costs one host memory read."""
    m = _STATUS_MIRRORS.get((dev.type, dev.index))
    if m is None or m["value"].value == 0:
        return
    torch.cuda.synchronize(dev)
    code = int(status_word(dev).item())
    status_word(dev).zero_()
    m["host"].zero_()
    torch.cuda.synchronize(dev)
    raise RuntimeError(f"an earlier tensor-core kernel on {dev} gave up on a device-side wait "
                       f"(code {code}): {status_string(-5)}; its outputs and those of later "
                       "launches are not valid")


_MIRROR_EVERY = 1           # launches after a kernel that gave up until the host copy of the word is set


def _on(dev: torch.device):
    """Make dev the current device for a library call; free when it already is."""
    if torch.cuda.current_device() == dev.index:
        return contextlib.nullcontext()
    return torch.cuda.device(dev)


def _capturing(dev: torch.device) -> bool:
    """Whether dev's current stream records a graph instead of running."""
    with _on(dev):
        return torch.cuda.is_current_stream_capturing()


_INDEX_CODES = {71: "sddmm", 72: "spmm", 73: "fused"}


def check_indices(dev, on: bool = True) -> None:
    """Checked-index mode of the CUDA-core kernels: columns derived from the metadata are clamped to
    [0, n_cols) and a code (71 SDDMM, 72 SpMM, 73 fused) is left in the device's status word, which
    check_status_word() reads.  SPLAT_B200_DEBUG switches it on for every CUDA-core launch."""
    dev = resolve_device(dev)
    check(_lib.splat_debug_check_indices(status_word(dev).data_ptr() if on else None),
          "splat_debug_check_indices")


def _debug_before(dev) -> bool:
    if not os.environ.get("SPLAT_B200_DEBUG"):
        return False
    check_indices(dev, True)
    return True


def check_status_word(dev) -> None:
    """Synchronises the device; raises if a band kernel reported a timed-out wait (and clears it)."""
    dev = resolve_device(dev)
    w = status_word(dev)
    code = int(w.item())
    if code != 0:
        w.zero_()
        m = _STATUS_MIRRORS.get((dev.type, dev.index))
        if m is not None:
            torch.cuda.synchronize(dev)
            m["host"].zero_()
        if code in _INDEX_CODES:
            raise RuntimeError(f"checked-index mode: a column derived from the row metadata lies outside "
                               f"[0, n_cols) in the {_INDEX_CODES[code]} kernel (code {code})")
        raise RuntimeError(f"band kernel gave up on a device-side wait (code {code}): "
                           f"{status_string(-5)}")


# ----------------------------------------------------------------------------------------------
# operators
# ----------------------------------------------------------------------------------------------
def _flat_bh(t: torch.Tensor, name: str):
    """(B, H, X, Y) tensor whose (B, H) dims collapse -> (bh, stride_bh, stride_x, stride_y)."""
    if t.dim() != 4:
        raise ValueError(f"{name} must be 4-dimensional (batch, heads, ., .)")
    B, H = t.shape[0], t.shape[1]
    sb, sh, sx, sy = t.stride()
    if B > 1 and H > 1 and sb != H * sh:
        raise ValueError(f"{name}: batch and head dimensions must be collapsible (stride {t.stride()})")
    stride_bh = sh if H > 1 else (sb if B > 1 else t.shape[2] * t.shape[3])
    return B * H, stride_bh, sx, sy


def _contig(t: torch.Tensor, name: str) -> torch.Tensor:
    if not t.is_contiguous():
        raise ValueError(f"{name} must be contiguous")
    return t


ERR_UNSUPPORTED_SHAPE, ERR_MISALIGNED, ERR_DRIVER = -6, -3, -7
# statuses of a tensor-core entry point that mean "this path does not apply, use the general one"
_BAND_NOT_APPLICABLE = (ERR_UNSUPPORTED_SHAPE, ERR_MISALIGNED, ERR_DRIVER)
_warned_cuda_core_16bit = False


def _warn_cuda_core_16bit(what: str) -> None:
    """16-bit operands that land on the CUDA-core kernels run many times slower than on the
    tensor-core path; say so once."""
    global _warned_cuda_core_16bit
    if not _warned_cuda_core_16bit:
        _warned_cuda_core_16bit = True
        import warnings
        warnings.warn(f"{what}: 16-bit operands are running on the CUDA-core kernels (pattern, layout, "
                      "alignment or head size outside what the tensor-core kernels take); expect a "
                      "much lower rate", RuntimeWarning, stacklevel=3)


def _band_candidate(x: torch.Tensor, path: int) -> bool:
    """The tensor-core kernels take 16-bit operands (of any d that is a multiple of 8 up to 128; the library checks
    that and the rest)."""
    return path != PATH_GENERIC and x.dtype in (torch.float16, torch.bfloat16) and x.numel() > 0


def _may_give_up(x: torch.Tensor, path: int) -> bool:
    """A tensor-core kernel may run: 16-bit operands, or fp32 bands (attention_split.cu, ops_split.cu)."""
    return _band_candidate(x, path) or (path == PATH_AUTO and x.dtype == torch.float32)


def _native_from_now_on(dev: torch.device) -> None:
    """The native path takes ordinary operands once the status word exists.  Setting it up synchronises, which a
    capture does not allow; the kernels without bounded waits need none."""
    if not _capturing(dev):
        status_word(dev)


def _plan_unless_captured(sTod_lin, sTod_tr, nnzs):
    """classify(), or None where a capture forbids to look at metadata that are new."""
    if _known_plan(sTod_lin, sTod_tr, nnzs) is None and _capturing(nnzs.device):
        return None
    return classify(sTod_lin, sTod_tr, nnzs)


def _rows_of_k(kt, plan, n_rows: int):
    """What the native path does with a 16-bit K^T that the tensor-core kernels cannot fetch: the row-major copy to
    work with, or None (not needed, no band pattern, no memory)."""
    with _on(kt.device):
        return _host.rows_of_k(kt, tuple(plan), n_rows)


def sddmm(x, y, output, sTod_lin, sTod_tr, nnzs, trailing_dim: int, path: int = PATH_AUTO) -> None:
    if _host.sddmm(x, y, output, sTod_lin, sTod_tr, nnzs, trailing_dim, path):
        return
    dev = x.device
    _native_from_now_on(dev)
    _contig(x, "x"); _contig(output, "output")
    B, H, L, d = x.shape
    bh, ksb, ksk, ksc = _flat_bh(y, "y")          # y is (B, H, d, n): dim 2 = k, dim 3 = column
    n_cols = y.shape[3]
    if y.shape[2] != d or bh != B * H or y.dtype != x.dtype or output.dtype != x.dtype:
        raise ValueError("sddmm: inconsistent operand shapes or dtypes")
    if tuple(output.shape) != (B, H, L, trailing_dim):
        raise ValueError(f"sddmm: output must have shape {(B, H, L, trailing_dim)}")
    # K layouts the tensor-core kernel reads: the transposed view of a contiguous (B,H,L,d) tensor, or
    # the reference's contiguous (B,H,d,L) K^T (the library checks the rest)
    k_layout_ok = ksb == n_cols * d and ((ksk == 1 and ksc == d) or (ksc == 1 and ksk == n_cols))
    if _band_candidate(x, path) and k_layout_ok:
        _raise_if_gave_up(dev)
        plan = classify(sTod_lin, sTod_tr, nnzs)
        plan_arr = (ctypes.c_int32 * 8)(*plan)
        rows = _rows_of_k(y, plan, L) if path == PATH_AUTO else None
        if rows is not None:
            y, ksb, ksk, ksc = rows, n_cols * d, 1, d
        with _on(dev):
            rc = _lib.splat_sddmm_band_table(x.data_ptr(), y.data_ptr(), ksb, ksc, ksk, output.data_ptr(),
                                       _f32_vec(sTod_lin, L, "sTod_lin"), _f32_vec(sTod_tr, L, "sTod_tr"),
                                       _f32_vec(nnzs, L, "nnzs"), bh, L, n_cols, d, trailing_dim,
                                       dtype_code(x.dtype), ctypes.cast(plan_arr, ctypes.c_void_p),
                                       band_table(sTod_lin, sTod_tr, nnzs, L), status_word(dev).data_ptr(), _stream(dev))
        if rc not in _BAND_NOT_APPLICABLE or path == PATH_BAND:
            check(rc, "splat_sddmm_band")
            if os.environ.get("SPLAT_B200_DEBUG"):
                check_status_word(dev)
            return
    if path == PATH_BAND:
        raise RuntimeError("sddmm: the band path does not apply to these operands")
    if x.dtype != torch.float32 and x.numel() > 0:
        _warn_cuda_core_16bit("sddmm")
    debug = _debug_before(dev)
    plan = None
    if x.dtype == torch.float32 and path == PATH_AUTO and x.numel() > 0:
        plan = _plan_unless_captured(sTod_lin, sTod_tr, nnzs)
    if plan is not None:
        _raise_if_gave_up(dev)             # (a tensor-core kernel may run: ops_split.cu)
        plan_arr = (ctypes.c_int32 * 8)(*plan)
        with _on(dev):
            rc = _lib.splat_sddmm_tile_status(x.data_ptr(), y.data_ptr(), ksb, ksc, ksk, output.data_ptr(),
                                              _f32_vec(sTod_lin, L, "sTod_lin"), _f32_vec(sTod_tr, L, "sTod_tr"),
                                              _f32_vec(nnzs, L, "nnzs"), bh, L, n_cols, d, trailing_dim,
                                              dtype_code(x.dtype), ctypes.cast(plan_arr, ctypes.c_void_p),
                                              status_word(dev).data_ptr(), _stream(dev))
        if rc not in _BAND_NOT_APPLICABLE:
            check(rc, "splat_sddmm_tile_status")
            return
    with _on(dev):
        check(_lib.splat_sddmm(x.data_ptr(), y.data_ptr(), ksb, ksc, ksk, output.data_ptr(),
                               _f32_vec(sTod_lin, L, "sTod_lin"), _f32_vec(sTod_tr, L, "sTod_tr"),
                               _f32_vec(nnzs, L, "nnzs"), bh, L, n_cols, d, trailing_dim,
                               dtype_code(x.dtype), _stream(dev)), "splat_sddmm")
    if debug:
        check_status_word(dev)


def softmax(x, output, nnzs, trailing_dim: int, scale: float = 1.0) -> None:
    if _host.softmax(x, output, nnzs, trailing_dim, scale):
        return
    dev = x.device
    _native_from_now_on(dev)
    _contig(x, "x"); _contig(output, "output")
    B, H, L, T = x.shape
    if T != trailing_dim or output.shape != x.shape or output.dtype != x.dtype:
        raise ValueError("softmax: inconsistent operand shapes or dtypes")
    with _on(dev):
        check(_lib.splat_softmax(x.data_ptr(), output.data_ptr(), _f32_vec(nnzs, L, "nnzs"), B * H,
                                 L, T, float(scale), dtype_code(x.dtype), _stream(dev)),
              "splat_softmax")


def spmm(x, y, output, sTod_lin, sTod_tr, nnzs, trailing_dim: int, path: int = PATH_AUTO) -> None:
    if _host.spmm(x, y, output, sTod_lin, sTod_tr, nnzs, trailing_dim, path):
        return
    dev = x.device
    _native_from_now_on(dev)
    _contig(x, "x"); _contig(y, "y"); _contig(output, "output")
    B, H, L, T = x.shape
    n_cols, d = y.shape[2], y.shape[3]
    if T != trailing_dim or tuple(output.shape) != (B, H, L, d) or y.dtype != x.dtype or \
            output.dtype != x.dtype or y.shape[:2] != x.shape[:2]:
        raise ValueError("spmm: inconsistent operand shapes or dtypes")
    if _band_candidate(x, path):
        _raise_if_gave_up(dev)
        plan_arr = (ctypes.c_int32 * 8)(*classify(sTod_lin, sTod_tr, nnzs))
        with _on(dev):
            rc = _lib.splat_spmm_band_table(x.data_ptr(), y.data_ptr(), output.data_ptr(),
                                      _f32_vec(sTod_lin, L, "sTod_lin"), _f32_vec(sTod_tr, L, "sTod_tr"),
                                      _f32_vec(nnzs, L, "nnzs"), B * H, L, n_cols, d, T,
                                      dtype_code(x.dtype), ctypes.cast(plan_arr, ctypes.c_void_p),
                                      band_table(sTod_lin, sTod_tr, nnzs, L), status_word(dev).data_ptr(), _stream(dev))
        if rc not in _BAND_NOT_APPLICABLE or path == PATH_BAND:
            check(rc, "splat_spmm_band")
            if os.environ.get("SPLAT_B200_DEBUG"):
                check_status_word(dev)
            return
    if path == PATH_BAND:
        raise RuntimeError("spmm: the band path does not apply to these operands")
    if x.dtype != torch.float32 and x.numel() > 0:
        _warn_cuda_core_16bit("spmm")
    debug = _debug_before(dev)
    plan = None
    if x.dtype == torch.float32 and path == PATH_AUTO and x.numel() > 0:
        plan = _plan_unless_captured(sTod_lin, sTod_tr, nnzs)
    if plan is not None:
        _raise_if_gave_up(dev)             # (a tensor-core kernel may run: ops_split.cu)
        plan_arr = (ctypes.c_int32 * 8)(*plan)
        with _on(dev):
            rc = _lib.splat_spmm_tile_status(x.data_ptr(), y.data_ptr(), output.data_ptr(),
                                             _f32_vec(sTod_lin, L, "sTod_lin"), _f32_vec(sTod_tr, L, "sTod_tr"),
                                             _f32_vec(nnzs, L, "nnzs"), B * H, L, n_cols, d, T,
                                             dtype_code(x.dtype), ctypes.cast(plan_arr, ctypes.c_void_p),
                                             status_word(dev).data_ptr(), _stream(dev))
        if rc not in _BAND_NOT_APPLICABLE:
            check(rc, "splat_spmm_tile_status")
            return
    with _on(dev):
        check(_lib.splat_spmm(x.data_ptr(), y.data_ptr(), output.data_ptr(),
                              _f32_vec(sTod_lin, L, "sTod_lin"), _f32_vec(sTod_tr, L, "sTod_tr"),
                              _f32_vec(nnzs, L, "nnzs"), B * H, L, n_cols, d, T,
                              dtype_code(x.dtype), _stream(dev)), "splat_spmm")
    if debug:
        check_status_word(dev)


def attention_fused(q, kt, v, output, sTod_lin, sTod_tr, nnzs, scale: float = 1.0,
                    path: int = PATH_AUTO, plan=None, lse=None) -> None:
    """q, v, output (B,H,L,d) contiguous; kt (B,H,d,L) -- contiguous (the reference's layout), or
    the transposed view of a contiguous (B,H,L,d) tensor.  The tensor-core path takes both (the
    contiguous one for stride-1 patterns).  lse: optional contiguous float32 (B,H,L) tensor that
    receives each row's log-sum-exp of the scaled scores (natural log, -inf for empty rows)."""
    dev = q.device
    _contig(q, "q"); _contig(v, "v"); _contig(output, "output")
    B, H, L, d = q.shape
    bh, ksb, ksk, ksc = _flat_bh(kt, "kt")
    n_cols = kt.shape[3]
    if kt.shape[2] != d or tuple(v.shape) != (B, H, n_cols, d) or output.shape != q.shape or \
            len({q.dtype, kt.dtype, v.dtype, output.dtype}) != 1:
        raise ValueError("attention: inconsistent operand shapes or dtypes")
    if lse is not None and (lse.dtype != torch.float32 or tuple(lse.shape) != (B, H, L) or
                            not lse.is_contiguous() or lse.device != dev):
        raise ValueError("attention: lse must be a contiguous float32 (B, H, L) tensor on the operands' device")
    plan_arr = None
    tensor_core = _band_candidate(q, path)      # a tensor-core kernel may run (the library decides)
    if path != PATH_GENERIC:
        if plan is None:
            plan = classify(sTod_lin, sTod_tr, nnzs)
        plan_arr = (ctypes.c_int32 * 8)(*plan)
    if _may_give_up(q, path):
        _raise_if_gave_up(dev)
    if tensor_core:
        rows = _rows_of_k(kt, plan, L) if path == PATH_AUTO else None
        if rows is not None:
            kt, ksb, ksk, ksc = rows, n_cols * d, 1, d
    sw = status_word(dev)
    table = band_table(sTod_lin, sTod_tr, nnzs, L) if tensor_core else None
    ran = ctypes.c_int32(0)
    _debug_before(dev)
    with _on(dev):
        check(_lib.splat_attention_fused_table(
            q.data_ptr(), kt.data_ptr(), ksb, ksc, ksk, v.data_ptr(), output.data_ptr(),
            lse.data_ptr() if lse is not None and lse.numel() > 0 else None,
            _f32_vec(sTod_lin, L, "sTod_lin"), _f32_vec(sTod_tr, L, "sTod_tr"),
            _f32_vec(nnzs, L, "nnzs"), bh, L, n_cols, d, float(scale), dtype_code(q.dtype),
            int(path), ctypes.cast(plan_arr, _vp) if plan_arr is not None else None,
            table, sw.data_ptr(), ctypes.byref(ran), _stream(dev)),
            "splat_attention_fused_table")
    if ran.value != PATH_BAND and q.dtype != torch.float32 and q.numel() > 0 and path == PATH_AUTO:
        _warn_cuda_core_16bit("attention")
    if os.environ.get("SPLAT_B200_DEBUG"):
        check_status_word(dev)


def module_forward(attributes: dict, x):
    """The fused call of a RegularAttention, from its __dict__ and [q, k^T, v]: the output tensor, or None
    when attention_fused() has to look at the operands (unusual ones, wrong ones, debug mode)."""
    return _host.module_forward(attributes, x)


_host.bind(*(ctypes.cast(getattr(_lib, name), _vp).value for name in (
    "splat_attention_fused_table", "splat_sddmm_band_table", "splat_spmm_band_table", "splat_sddmm_tile_status",
    "splat_spmm_tile_status",
    "splat_softmax", "splat_acsr_from_mask_u8", "splat_transpose_16", "splat_sddmm", "splat_spmm")), _warn_cuda_core_16bit)
