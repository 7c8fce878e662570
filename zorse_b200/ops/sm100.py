"""ctypes bindings of the hand-written sm_100a kernels (`csrc/`, built by `ops/build.py`).

Every function here launches one of this repository's own CUDA kernels on the current
torch stream; there is no fallback: if the library is missing on a machine with a GPU
the import of the library raises.  Tensors are passed as raw device pointers.

`launch_count()` counts the kernels launched through this module (bench.py reports it).
"""
from __future__ import annotations

import ctypes
import functools
import math
import os
import warnings
from ctypes import c_float, c_int, c_long, c_void_p
from pathlib import Path
from typing import Optional

import torch

_LIB_PATH = Path(__file__).resolve().parents[1] / "_C" / "libzorse_sm100.so"
_lib = None
_launches = 0
_status: dict[int, torch.Tensor] = {}

GEMM_OUT_F32 = 1
GEMM_ACCUMULATE = 2
GEMM_GELU = 4
GEMM_RELU = 8

GEMM_KERNEL = os.environ.get("ZORSE_GEMM", "2cta")

ACT_GELU_TANH = 0
ACT_RELU = 1
ACT_GELU_ERF = 2


# Argument types of the entry points a training step calls all the time, in order (p pointer, i int, l long, f float):
# with them ctypes converts plain Python numbers itself, which is cheaper than a c_int / c_void_p object per argument.
_SIGNATURES = {
    "zb_gemm2_bf16": "pppiiiiiiiippiiipp",
    "zb_gemm2_split_bf16": "pppiiiiiiiippiiplpp", "zb_gemm_bf16": "pppiiiiiiiippiiiipp",
    "zb_norm_fwd": "pppppiifip", "zb_norm_fwd2": "pppppiifip",
    "zb_norm_bwd": "ppppppppppiiiiip", "zb_norm_bwd2": "ppppppppppiiiiip",
    "zb_colsum": "piiippiip", "zb_rope": "ppiiiiiip", "zb_swiglu_fwd": "pplip", "zb_swiglu_bwd": "ppplip",
    "zb_act_fwd": "pplip", "zb_act_bwd": "ppplip", "zb_embedding_fwd": "ppppiiiiip", "zb_embedding_bwd": "ppppiiiiiip",
    "zb_cross_entropy": "ppppiilflp", "zb_adam": "ppppplfffffifiip",
    "zb_flash_fwd": "pppiiiiiiifipp", "zb_flash_fwd2": "pppiiiiiiifipp",
    "zb_flash_fwd4": "pppiiiiiiifipipip", "zb_flash_bwd3": "ppppppiiiiiiifpipip",
}
_CTYPES = {"p": c_void_p, "i": c_int, "l": c_long, "f": c_float}


class KernelError(RuntimeError):
    pass


def available() -> bool:
    return _LIB_PATH.exists()


def lib():
    """Loads (building if needed) the kernel library. Raises if it cannot be had."""
    global _lib
    if _lib is None:
        path = _LIB_PATH
        if os.environ.get("ZORSE_DEBUG_BOUNDS", "0") == "1":
            # the checking build: same entry points, kernels verify their indices (see csrc/common/ptx.cuh)
            from . import build as _build

            path = _build.build(debug_bounds=True)
        elif not path.exists():
            from . import build as _build

            _build.build()
        _lib = ctypes.CDLL(str(path))
        _lib.zb_last_error.restype = ctypes.c_char_p
        for name, sig in _SIGNATURES.items():
            getattr(_lib, name).argtypes = [_CTYPES[c] for c in sig]
        if "ZORSE_RS_ADAM_VARIANT" in os.environ:      # 0 / 1 select a peer-load kernel (1 is the library default)
            _lib.zb_set_rs_adam_variant(c_int(int(os.environ["ZORSE_RS_ADAM_VARIANT"])))
        _load_fast()
    return _lib


# The module csrc/host/fastops.cpp: the same entry points for the calls of a training step, without Python in between.  It
# answers None to arguments it was not written for; the wrappers below take those.  None until the library is loaded, and where
# there is neither a module for this torch nor a way to build it (an installed copy): the wrappers then take every call.
_fast = None
_FAST_ENTRIES = ("zb_gemm_bf16", "zb_gemm2_bf16", "zb_gemm2_split_bf16", "zb_gemm2_workspace", "zb_norm_fwd", "zb_norm_bwd2",
                 "zb_norm_bwd2_rows", "zb_colsum", "zb_rope", "zb_swiglu_fwd", "zb_swiglu_bwd", "zb_act_fwd", "zb_act_bwd",
                 "zb_flash_fwd4", "zb_flash_bwd3", "zb_flash_bwd2_stats_floats", "zb_gemm2_act_fwd",
                 "zb_gemm2_act_bwd", "zb_gemm2_rope_fwd", "zb_column_sums", "zb_last_error")   # the order of its `Entry`


def _load_fast() -> None:
    global _fast
    import importlib.util

    from . import build as _build

    try:
        path = _build.build_fast()
    except _build.FastModuleUnavailable as e:
        warnings.warn(f"no native call module, every launch goes through Python: {e}", RuntimeWarning, stacklevel=2)
        return
    spec = importlib.util.spec_from_file_location("zorse_fastops", path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    mod.init(tuple(ctypes.cast(getattr(_lib, n), c_void_p).value for n in _FAST_ENTRIES), KernelError)
    for dev, word in _status.items():
        mod.set_status(dev, word.data_ptr())
    _fast = mod


def launch_count() -> int:
    return _launches + (_fast.launch_count() if _fast is not None else 0)


def _stream() -> c_void_p:
    # the raw handle: building a torch.cuda.Stream object for it costs a quarter of a launch's host time
    return c_void_p(torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice()))


def _p(t: Optional[torch.Tensor]) -> c_void_p:
    return c_void_p(0 if t is None else t.data_ptr())


def _a(t: Optional[torch.Tensor]) -> int:
    """Device address for an entry point listed in _SIGNATURES (a plain int: no other may take it)."""
    return 0 if t is None else t.data_ptr()


def status_word(device=None) -> torch.Tensor:
    """Device int32 that kernels write a non-zero code to when a bounded wait runs out."""
    if isinstance(device, torch.device):
        dev = device.index
    else:
        dev = torch.cuda.current_device() if device is None else torch.device(device).index
    if dev not in _status:
        _status[dev] = torch.zeros(1, dtype=torch.int32, device=f"cuda:{dev}")
        if _fast is not None:
            _fast.set_status(dev, _status[dev].data_ptr())
    return _status[dev]


_STATUS_NAMES = {
    1: "TMA stage never landed", 2: "stage never released", 3: "accumulator never completed",
    4: "accumulator never drained", 5: "flag wait ran out", 6: "bad argument", 7: "wait ran out",
}


_BOUNDS_SITES = {1: "GEMM tile origin", 2: "GEMM epilogue row / column", 3: "all-gather chunk", 4: "all-gather flag index",
                 5: "optimizer slice", 8: "attention tile"}


def check_status(device=None) -> None:
    """Synchronising read of the status word; raises KernelError if a kernel gave up."""
    raise_status(int(status_word(device).item()), device)


def raise_status(v: int, device=None) -> None:
    """Raises KernelError if `v`, a value read from the device's status word, says that a kernel gave up (the word is cleared)."""
    if v != 0:
        status_word(device).zero_()
        code = v & 0xf
        if code == 8:
            site = (v >> 4) & 0xf
            raise KernelError(f"sm100 kernel (checking build) found an index outside its tensor: site {site} "
                              f"({_BOUNDS_SITES.get(site, '?')}) in block {v >> 8}; the access was skipped")
        raise KernelError(
            f"sm100 kernel reported status {v & 0xff} ({_STATUS_NAMES.get(v & 0xff, '?')}) in block {v >> 8}")


def _check(rc: int, what: str) -> None:
    global _launches
    if rc != 0:
        raise KernelError(f"{what}: {lib().zb_last_error().decode()}")
    _launches += 1


def _bf16(t: torch.Tensor, name: str) -> None:
    if t.dtype != torch.bfloat16 or not t.is_cuda:
        raise TypeError(f"{name} must be a CUDA bf16 tensor, got {t.dtype} on {t.device}")


# --------------------------------------------------------------------------- GEMM
@functools.lru_cache(maxsize=4096)
def _gemm2_workspace(M: int, N: int, K: int, device: int) -> int:
    """Bytes of workspace the pair kernel wants for this product (a function of the sizes and of the number of SMs of the
    current device, whose index is `device`, as the operands' is), 0 for none."""
    return lib().zb_gemm2_workspace(c_int(M), c_int(N), c_int(K))


def gemm(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor, *, a_mn: bool = False, b_mn: bool = False,
         bias: Optional[torch.Tensor] = None, addend: Optional[torch.Tensor] = None, accumulate: bool = False,
         act: Optional[str] = None, bn: int = 0, max_ctas: int = 0, kernel: Optional[str] = None) -> torch.Tensor:
    """out[M,N] = A @ B^T (+bias) (+addend), or out += ... with accumulate.

    a: [M,K] (K-major) or [K,M] when a_mn; b: [N,K] (K-major) or [K,N] when b_mn.
    out: bf16 or fp32 [M,N]. kernel: "1cta" (128x{128,256} tile per CTA), "2cta" (256x256 tile per
    CTA pair, tcgen05 cta_group::2), "2cta_accpf" (another name of "2cta", whose epilogue requests the old C tile of a
    bf16 `accumulate` ahead of the accumulators) or None = GEMM_KERNEL default ("2cta" for M, N >= 256).
    """
    _bf16(a, "a"); _bf16(b, "b")
    # shapes, strides and types are read once each: this function runs for every product of a step
    M, N = out.shape
    (rows_a, cols_a), (rows_b, cols_b) = a.shape, b.shape
    K = rows_a if a_mn else cols_a
    assert (cols_a if a_mn else rows_a) == M, (a.shape, out.shape, a_mn)
    assert (rows_b == K and cols_b == N) if b_mn else (rows_b == N and cols_b == K), (b.shape, (N, K), b_mn)
    (lda, step_a), (ldb, step_b), (ldc, step_c) = a.stride(), b.stride(), out.stride()
    assert step_a == 1 and step_b == 1 and step_c == 1
    flags, dtype = 0, out.dtype
    if dtype == torch.float32:
        flags |= GEMM_OUT_F32
    elif dtype != torch.bfloat16:
        raise TypeError("gemm output must be bf16 or fp32")
    if accumulate:
        flags |= GEMM_ACCUMULATE
    if act == "gelu":
        flags |= GEMM_GELU
    elif act == "relu":
        flags |= GEMM_RELU
    kern = kernel or GEMM_KERNEL
    if kern in ("2cta", "2cta_accpf") and bn == 0 and M >= 256 and N >= 256:
        # a long reduction whose last wave of tiles would leave most of the GPU idle is cut up there (below this length
        # it never is: see the kernel's plan)
        ws_bytes = _gemm2_workspace(M, N, K, a.device.index) if K > 3000 and max_ctas == 0 else 0
        if ws_bytes:
            ws = torch.empty(ws_bytes, dtype=torch.uint8, device=a.device)
            rc = lib().zb_gemm2_split_bf16(_a(a), _a(b), _a(out), M, N, K, lda, ldb, ldc,
                                           int(a_mn), int(b_mn), _a(bias), _a(addend),
                                           0 if addend is None else addend.stride(0), flags, _a(ws), ws_bytes,
                                           _a(status_word(a.device)), _stream())
            _check(rc, "gemm2_split")
            return out
        rc = lib().zb_gemm2_bf16(_a(a), _a(b), _a(out), M, N, K, lda, ldb, ldc, int(a_mn), int(b_mn),
                                 _a(bias), _a(addend), 0 if addend is None else addend.stride(0),
                                 flags, max_ctas, _a(status_word(a.device)), _stream())
        _check(rc, "gemm2")
        return out
    rc = lib().zb_gemm_bf16(_a(a), _a(b), _a(out), M, N, K, lda, ldb, ldc, int(a_mn), int(b_mn),
                            _a(bias), _a(addend), 0 if addend is None else addend.stride(0),
                            flags, bn, max_ctas, _a(status_word(a.device)), _stream())
    _check(rc, "gemm")
    return out


# --------------------------------------------------------------------------- norms
NORM_FWD_VERSION = int(os.environ.get("ZORSE_NORM_FWD", "1"))


def norm_fwd(x, w, b, eps: float, layernorm: bool, version: Optional[int] = None):
    """version 1: one CTA per row; version 2 (candidate): one warp per row, no block barriers."""
    _bf16(x, "x")
    T, H = x.shape
    y = torch.empty_like(x)
    stats = torch.empty(T, 2, dtype=torch.float32, device=x.device)
    fn = lib().zb_norm_fwd2 if (version or NORM_FWD_VERSION) == 2 else lib().zb_norm_fwd
    _check(fn(_a(x), _a(w), _a(b), _a(y), _a(stats), T, H, eps,
              int(layernorm), _stream()), "norm_fwd")
    return y, stats


NORM_BWD_VERSION = int(os.environ.get("ZORSE_NORM_BWD", "2"))


def norm_bwd(dy, x, w, stats, dres, dw, db, layernorm: bool, accumulate: bool = True, version: Optional[int] = None):
    """Returns dx (+dres). dw/db: gradient slots (fp32 or bf16) accumulated into.
    version 2: next-row prefetch, one barrier per row, parallel column reduction."""
    T, H = x.shape
    dx = torch.empty_like(x)
    P = lib().zb_norm_partial_rows(c_int(T))
    part_dw = torch.empty(P, H, dtype=torch.float32, device=x.device)
    part_db = torch.empty(P, H, dtype=torch.float32, device=x.device) if (layernorm and db is not None) else None
    gf32 = int(dw.dtype == torch.float32)
    fn = lib().zb_norm_bwd2 if (version or NORM_BWD_VERSION) == 2 else lib().zb_norm_bwd
    _check(fn(_a(dy), _a(x), _a(w), _a(stats), _a(dres), _a(dx), _a(part_dw), _a(part_db),
                             _a(dw), _a(db), T, H, int(layernorm), gf32,
                             int(accumulate), _stream()), "norm_bwd")
    return dx


def colsum_accumulate(dy, out, accumulate: bool = True):
    """out[n] (+)= sum_t dy[t, n] (bias gradients)."""
    T, N = dy.shape
    part = torch.empty(min(T, 64), N, dtype=torch.float32, device=dy.device)
    _check(lib().zb_colsum(_a(dy), T, N, dy.stride(0), _a(part), _a(out),
                           int(out.dtype == torch.float32), int(accumulate), _stream()), "colsum")
    return out


# --------------------------------------------------------------------------- elementwise
def rope_(buf, cs, S: int, nheads: int, d: int, backward: bool = False):
    """In-place rotate-half RoPE on heads [0, nheads) of a packed [T, width] buffer."""
    T = buf.shape[0]
    _check(lib().zb_rope(_a(buf), _a(cs), T, S, nheads, d, buf.stride(0),
                         int(backward), _stream()), "rope")
    return buf


def swiglu_fwd(gu):
    T, F2 = gu.shape
    out = torch.empty(T, F2 // 2, dtype=gu.dtype, device=gu.device)
    _check(lib().zb_swiglu_fwd(_a(gu), _a(out), T, F2 // 2, _stream()), "swiglu_fwd")
    return out


def swiglu_bwd(gu, dout):
    dgu = torch.empty_like(gu)
    T, F2 = gu.shape
    _check(lib().zb_swiglu_bwd(_a(gu), _a(dout), _a(dgu), T, F2 // 2, _stream()), "swiglu_bwd")
    return dgu


def act_fwd(x, kind: int):
    y = torch.empty_like(x)
    _check(lib().zb_act_fwd(_a(x), _a(y), x.numel(), kind, _stream()), "act_fwd")
    return y


def act_bwd(x, dy, kind: int):
    dx = torch.empty_like(x)
    _check(lib().zb_act_bwd(_a(x), _a(dy), _a(dx), x.numel(), kind, _stream()), "act_bwd")
    return dx


def patches(img, patch: int, kdim: int):
    """Non-overlapping patches of fp32 images [B, C, H, W] as bf16 rows [B * patches, kdim] (channel, row, column within
    the patch; zeros behind C * patch^2)."""
    if img.dtype != torch.float32 or not img.is_cuda:
        raise TypeError(f"patches needs a CUDA fp32 tensor, got {img.dtype} on {img.device}")
    img = img.contiguous()
    B, C, H, W = img.shape
    out = torch.empty(B * (H // patch) * (W // patch), kdim, dtype=torch.bfloat16, device=img.device)
    _check(lib().zb_patches(_p(img), _p(out), c_int(B), c_int(C), c_int(H), c_int(W), c_int(patch), c_int(kdim),
                            _stream()), "patches")
    return out


def embedding_fwd(ids, table, pos_table=None, S: int = 1, pos_offset: int = 0):
    T = ids.numel()
    V, H = table.shape
    out = torch.empty(T, H, dtype=table.dtype, device=table.device)
    _check(lib().zb_embedding_fwd(_a(ids), _a(table), _a(pos_table), _a(out), T, H, V,
                                  S, pos_offset, _stream()), "embedding_fwd")
    return out


def embedding_bwd(ids, dout, dtable, dpos=None, S: int = 1, pos_offset: int = 0):
    T = ids.numel()
    V, H = dtable.shape
    _check(lib().zb_embedding_bwd(_a(ids), _a(dout), _a(dtable), _a(dpos), T, H, V,
                                  S, pos_offset, int(dtable.dtype == torch.float32),
                                  _stream()), "embedding_bwd")


# --------------------------------------------------------------------------- loss
def cross_entropy(logits, targets, grad_scale: float, dlogits=None, ignore_index: int = -100):
    """Returns per-row losses (fp32). Writes d(loss)/d(logits) * grad_scale into dlogits
    (may alias logits) when given."""
    T, V = logits.shape
    loss_rows = torch.empty(T, dtype=torch.float32, device=logits.device)
    _check(lib().zb_cross_entropy(_a(logits), _a(targets), _a(dlogits), _a(loss_rows), T, V,
                                  logits.stride(0), grad_scale, ignore_index,
                                  _stream()), "cross_entropy")
    return loss_rows


# --------------------------------------------------------------------------- optimizer
def adam_step(p, m, v, g, p16, *, lr, beta1, beta2, eps, weight_decay, step, grad_scale=1.0, zero_grad=False):
    n = p.numel()
    _check(lib().zb_adam(_a(p), _a(m), _a(v), _a(g), _a(p16), n, lr, beta1,
                         beta2, eps, weight_decay, step, grad_scale,
                         int(g.dtype == torch.float32), int(zero_grad), _stream()), "adam")


# --------------------------------------------------------------------------- attention
def _window(window: int, S: int) -> int:
    """0 (none) for a window no shorter than the sequence: every earlier key is visible, and the kernels' 32-bit tile bounds
    (key + window and the like) stay far from their limit."""
    return 0 if window >= S else window


# 1 / 2 / 4 force a version.  0: the op layer (`api.Sm100Ops`, what layers call) takes version 4 (two query tiles per CTA,
# 256 query rows) at every size; `flash_fwd` called without a version takes it, or version 1 (one 128-row tile per CTA) for
# small problems.
ATTN_FWD_VERSION = int(os.environ.get("ZORSE_ATTN_FWD", "0"))


ATTN_FWD4_FLAGS = int(os.environ.get("ZORSE_ATTN_FWD4_FLAGS", "1"))


def _auto_fwd_version(B: int, S: int, Hq: int, D: int) -> int:
    # the two-tile kernel where it fills the GPU (d = 64) or nearly half of it (d = 128)
    return 4 if B * Hq * ((S + 255) // 256) >= (64 if D == 128 else 148) else 1


def flash_fwd(qkv, B: int, S: int, Hq: int, Hkv: int, D: int, causal: bool = True, window: int = 0,
              scale: Optional[float] = None, version: Optional[int] = None, flags: Optional[int] = None,
              trace: Optional[torch.Tensor] = None, trace_ctas: int = 0):
    """qkv: packed [B*S, (Hq+2Hkv)*D]. Returns (out [B*S, Hq*D], lse [B, Hq, S]).
    version 1: one query tile per CTA, S double-buffered in TMEM, P staged through shared memory (default here
    for small problems); version 2: two query tiles per CTA, P kept in
    TMEM; version 4 (the op layer's, and default otherwise, 143 against 257 us on 32 heads of 4096 tokens, d = 128): two
    query tiles, one MMA issuer, score rows in registers (`flags` 1: two-wide
    fp32 math, 2: also a quarter of the exponentials as a polynomial on the fma pipe; `trace`: zeroed int64 buffer from `flash_fwd4_trace_buffer` for a phase timeline)."""
    _bf16(qkv, "qkv")
    assert qkv.shape == (B * S, (Hq + 2 * Hkv) * D) and qkv.is_contiguous()
    out = torch.empty(B * S, Hq * D, dtype=qkv.dtype, device=qkv.device)
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device=qkv.device)
    sc = (1.0 / math.sqrt(D)) if scale is None else scale
    window = _window(window, S)
    ver = version or ATTN_FWD_VERSION or _auto_fwd_version(B, S, Hq, D)
    if ver == 4:
        fl = ATTN_FWD4_FLAGS if flags is None else flags
        _check(lib().zb_flash_fwd4(_a(qkv), _a(out), _a(lse), B, S, Hq, Hkv, D,
                                   int(causal), window, sc, out.stride(0),
                                   _a(status_word(qkv.device)), fl, _a(trace),
                                   trace_ctas if trace is not None else 0, _stream()), "flash_fwd4")
        return out, lse
    fn = {1: lib().zb_flash_fwd, 2: lib().zb_flash_fwd2}[ver]
    _check(fn(_a(qkv), _a(out), _a(lse), B, S, Hq, Hkv, D,
                              int(causal), window, sc, out.stride(0),
                              _a(status_word(qkv.device)), _stream()), "flash_fwd")
    return out, lse


_attn_scratch2: dict = {}


def _flash_bwd2(do, qkv, o, lse, B, S, Hq, Hkv, D, causal, window, scale, trace, trace_ctas):
    key = (qkv.device.index, B, S, Hq, D)
    if key not in _attn_scratch2:
        n = lib().zb_flash_bwd2_stats_floats(c_int(B), c_int(S), c_int(Hq))
        # the accumulator is zeroed once: the kernel that converts it leaves it so
        _attn_scratch2[key] = (torch.zeros(n, dtype=torch.float32, device=qkv.device),
                               torch.zeros(B * S * Hq * D, dtype=torch.float32, device=qkv.device))
    stats, dq_acc = _attn_scratch2[key]
    dqkv = torch.empty_like(qkv)
    sc = (1.0 / math.sqrt(D)) if scale is None else scale
    _check(lib().zb_flash_bwd2(_p(do), _p(qkv), _p(o), _p(lse), _p(dqkv), _p(stats), _p(dq_acc), c_int(B), c_int(S),
                               c_int(Hq), c_int(Hkv), c_int(D), c_int(int(causal)), c_int(window), c_float(sc),
                               _p(status_word(qkv.device)), _p(trace), c_int(trace_ctas if trace is not None else 0),
                               _stream()), "flash_bwd2")
    global _launches
    _launches += 2  # statistics + finish kernels
    return dqkv


def _flash_bwd3(do, qkv, o, lse, B, S, Hq, Hkv, D, causal, window, scale, parts: int = 3, trace=None, trace_ctas: int = 0):
    key = (qkv.device.index, B, S, Hq)
    if key not in _attn_scratch3:
        n = lib().zb_flash_bwd2_stats_floats(c_int(B), c_int(S), c_int(Hq))
        _attn_scratch3[key] = torch.zeros(n, dtype=torch.float32, device=qkv.device)
    stats = _attn_scratch3[key]
    dqkv = torch.empty_like(qkv)
    sc = (1.0 / math.sqrt(D)) if scale is None else scale
    _check(lib().zb_flash_bwd3(_a(do), _a(qkv), _a(o), _a(lse), _a(dqkv), _a(stats), B, S, Hq,
                               Hkv, D, int(causal), window, sc,
                               _a(status_word(qkv.device)), parts, _a(trace),
                               trace_ctas if trace is not None else 0, _stream()), "flash_bwd3")
    global _launches
    _launches += 2  # statistics + the second main kernel
    return dqkv


_attn_scratch3: dict = {}


def flash_bwd2_trace_buffer(device, ctas: int) -> torch.Tensor:
    w, e = lib().zb_flash_bwd2_trace_warps(), lib().zb_flash_bwd2_trace_events()
    return torch.zeros(ctas, w, e, dtype=torch.int64, device=device)


def flash_fwd4_trace_buffer(device, ctas: int) -> torch.Tensor:
    """Zeroed event buffer [ctas, warps, events] for `flash_fwd(version=4, trace=...)`; an event is
    (clock64 << 8) | code, 0 = unused slot."""
    w, e = lib().zb_flash_fwd4_trace_warps(), lib().zb_flash_fwd4_trace_events()
    return torch.zeros(ctas, w, e, dtype=torch.int64, device=device)


_attn_scratch: dict = {}


# 0 = default = version 3 (two kernels, no atomics: 427 us for 32 heads of 4096 tokens, d = 128);
# 1 / 2 / 3 force a version
ATTN_BWD_VERSION = int(os.environ.get("ZORSE_ATTN_BWD", "0"))


def flash_bwd(do, qkv, o, lse, B: int, S: int, Hq: int, Hkv: int, D: int, causal: bool = True, window: int = 0,
              scale: Optional[float] = None, version: Optional[int] = None, trace: Optional[torch.Tensor] = None,
              trace_ctas: int = 0):
    """Returns dqkv packed like qkv. Scratch (fp32 dQ accumulator, delta) is cached per shape
    and device; the accumulator is left zeroed by the kernel that converts it to bf16.
    version 1: scores with queries on the TMEM lanes, P and dS staged through shared
    memory; version 2: transposed scores, P^T / dS^T consumed from tensor memory, two Q/dO stages
    (`trace`: zeroed buffer from `flash_bwd2_trace_buffer`); version 3 (default): two kernels without atomics, dK / dV per
    key tile and dQ per query tile (scores are formed twice; no fp32 dQ accumulator)."""
    _bf16(do, "do"); _bf16(qkv, "qkv")
    assert do.is_contiguous() and qkv.is_contiguous() and o.is_contiguous()
    window = _window(window, S)
    ver = version or ATTN_BWD_VERSION or 3
    if ver == 3:
        return _flash_bwd3(do, qkv, o, lse, B, S, Hq, Hkv, D, causal, window, scale, trace=trace, trace_ctas=trace_ctas)
    if ver == 2:
        return _flash_bwd2(do, qkv, o, lse, B, S, Hq, Hkv, D, causal, window, scale, trace, trace_ctas)
    key = (qkv.device.index, B, S, Hq, D)
    if key not in _attn_scratch:
        _attn_scratch[key] = (torch.empty(B * Hq * S, dtype=torch.float32, device=qkv.device),
                              torch.zeros(B * S * Hq * D, dtype=torch.float32, device=qkv.device))
    delta, dq_acc = _attn_scratch[key]
    dqkv = torch.empty_like(qkv)
    sc = (1.0 / math.sqrt(D)) if scale is None else scale
    _check(lib().zb_flash_bwd(_p(do), _p(qkv), _p(o), _p(lse), _p(dqkv), _p(delta), _p(dq_acc), c_int(B), c_int(S),
                              c_int(Hq), c_int(Hkv), c_int(D), c_int(int(causal)), c_int(window), c_float(sc),
                              _p(status_word(qkv.device)), _stream()), "flash_bwd")
    global _launches
    _launches += 2  # delta + finish kernels
    return dqkv


# --------------------------------------------------------------------------- fused collectives
def _ptr_array(ptrs):
    arr = (c_void_p * len(ptrs))(*[c_void_p(int(x)) for x in ptrs])
    return arr


def ag_gemm(a: torch.Tensor, full: torch.Tensor, w_offset: int, w_shape, out: torch.Tensor, *, shard_ptrs, R: int,
            r: int, shard_elems: int, chunk_bytes: int, chunk_flags: torch.Tensor, epoch: int,
            version_flags: torch.Tensor, need_version: int, bias=None, addend=None) -> torch.Tensor:
    """out = a @ W^T with W = full[w_offset : w_offset + N*K].view(N, K), while the same kernel
    pulls the other ranks' shards of the unit into `full` (all-gather fused with the GEMM).
    shard_ptrs: device addresses of every rank's bf16 shard (peer-mapped), by group rank."""
    _bf16(a, "a")
    N, K = w_shape
    M = a.shape[0]
    assert out.shape == (M, N) and a.shape[1] == K and out.dtype == torch.bfloat16
    # the 2-CTA core (256 x 256 tiles per CTA pair) when the problem has at least one such tile, like `gemm`
    two_cta = GEMM_KERNEL == "2cta" and M >= 256 and N >= 256 and os.environ.get("ZORSE_AG_GEMM", "2cta") != "1cta"
    fn = lib().zb_ag_gemm2_bf16 if two_cta else lib().zb_ag_gemm_bf16
    rc = fn(_p(a), _p(full), c_long(w_offset * 2), _p(out), c_int(M), c_int(N), c_int(K),
                               c_int(a.stride(0)), c_int(out.stride(0)), _p(bias), _p(addend),
                               c_int(0 if addend is None else addend.stride(0)), c_int(0), _ptr_array(shard_ptrs),
                               c_int(R), c_int(r), c_long(shard_elems * 2), c_int(chunk_bytes), _p(chunk_flags),
                               c_int(epoch), _p(version_flags), c_int(need_version), _p(status_word(a.device)),
                               _stream())
    _check(rc, "ag_gemm")
    return out


def gemm_rs(a: torch.Tensor, b: torch.Tensor, *, b_mn: bool, dst_ptrs, flag_ptrs, flag_index: int, epoch: int,
            counter: torch.Tensor, ldc: int, max_ctas: int = 0) -> None:
    """Partial product a @ b^T (b_mn: a @ b) whose rows are scattered for a row-wise reduce-scatter over
    R = len(dst_ptrs) processes: rows of chunk q are stored (bf16, row stride ldc) at dst_ptrs[q], a device
    address that may be in a peer's memory; afterwards `epoch` is stored to flag_ptrs[q][flag_index]."""
    _bf16(a, "a"); _bf16(b, "b")
    M, K = a.shape
    N = b.shape[1] if b_mn else b.shape[0]
    assert (b.shape[0] if b_mn else b.shape[1]) == K and a.stride(-1) == 1 and b.stride(-1) == 1
    R = len(dst_ptrs)
    rc = lib().zb_gemm2_rs_bf16(_p(a), _p(b), c_int(M), c_int(N), c_int(K), c_int(a.stride(0)), c_int(b.stride(0)),
                                c_int(ldc), c_int(int(b_mn)), _ptr_array(dst_ptrs), _ptr_array(flag_ptrs), c_int(R),
                                c_int(flag_index), c_int(epoch), _p(counter), c_int(max_ctas),
                                _p(status_word(a.device)), _stream())
    _check(rc, "gemm_rs")


def rs_finish(slots: torch.Tensor, flags: torch.Tensor, R: int, rows: int, H: int, epoch: int, out: torch.Tensor,
              resid: Optional[torch.Tensor] = None, bias: Optional[torch.Tensor] = None, wait_seconds: float = 2.0):
    """out[rows, H] = sum over the R staging slots ([R, rows, H] bf16, filled by the peers' gemm_rs) (+ resid)
    (+ bias), after every sender's flag has reached `epoch` (bounded wait)."""
    rc = lib().zb_rs_finish(_p(slots), _p(flags), c_int(R), c_int(rows), c_int(H), c_int(H), c_int(epoch), _p(resid),
                            c_int(0 if resid is None else resid.stride(0)), _p(bias), _p(out), c_int(out.stride(0)),
                            ctypes.c_double(wait_seconds), _p(status_word(out.device)), _stream())
    _check(rc, "rs_finish")
    return out


def tp_norm_push(*, w, b, eps: float, layernorm: bool, y_local, dst_ptrs, flag_ptrs, flag_index: int, epoch: int,
                 stats, counter, x=None, slots=None, in_flags=None, in_epoch: int = 0, resid=None, bias=None, h_out=None,
                 wait_seconds: float = 2.0) -> None:
    """Row-wise norm whose output also goes to every lane member's gathered buffer (dst_ptrs: device addresses
    of this process's row block there).  Input rows: `x`, or the sum of the reduce-scatter `slots`
    ([R, rows, H], ready when in_flags reach in_epoch) + resid + bias, which is written to h_out."""
    rows, H = y_local.shape
    R_in = 0 if slots is None else slots.numel() // (rows * H)
    rc = lib().zb_tp_norm_push(_p(x), _p(slots), _p(in_flags), c_int(R_in), c_int(in_epoch), _p(resid),
                               c_int(0 if resid is None else resid.stride(0)), _p(bias), _p(h_out), _p(w), _p(b),
                               c_float(eps), c_int(int(layernorm)), _p(y_local), _ptr_array(dst_ptrs),
                               _ptr_array(flag_ptrs), c_int(len(dst_ptrs)), c_int(flag_index), c_int(epoch), _p(stats),
                               c_int(rows), c_int(H), _p(counter), ctypes.c_double(wait_seconds),
                               _p(status_word(y_local.device)), _stream())
    _check(rc, "tp_norm_push")


def tp_push(src: torch.Tensor, dst_ptrs, flag_ptrs, flag_index: int, epoch: int, counter) -> None:
    """Copies the contiguous tensor `src` to every device address in dst_ptrs, then stores `epoch` to
    flag_ptrs[q][flag_index] (all-gather by stores, for rows that need no arithmetic)."""
    assert src.is_contiguous()
    rc = lib().zb_tp_push(_p(src), _ptr_array(dst_ptrs), _ptr_array(flag_ptrs), c_int(len(dst_ptrs)), c_int(flag_index),
                          c_int(epoch), c_long(src.numel() * src.element_size()), _p(counter),
                          _p(status_word(src.device)), _stream())
    _check(rc, "tp_push")


def rs_adam(grad_ptrs, flag_ptrs, R: int, r: int, shard_elems: int, master, m, v, p16, *, lr, beta1, beta2, eps,
            weight_decay, step, grad_scale, grad_f32: bool, epoch: int, counter: torch.Tensor, max_blocks: int = 0,
            wait_seconds: float = 2.0):
    """Fused reduce-scatter + Adam: sums slice r of every rank's gradient bucket (peer loads)
    and updates master/m/v/p16 in one pass. grad_ptrs / flag_ptrs: device addresses by group rank."""
    rc = lib().zb_rs_adam(_ptr_array(grad_ptrs), _ptr_array(flag_ptrs), c_int(R), c_int(r), c_long(shard_elems),
                          _p(master), _p(m), _p(v), _p(p16), c_float(lr), c_float(beta1), c_float(beta2), c_float(eps),
                          c_float(weight_decay), c_int(step), c_float(grad_scale), c_int(int(grad_f32)), c_int(epoch),
                          _p(counter), c_int(max_blocks), ctypes.c_double(wait_seconds),
                          _p(status_word(master.device)), _stream())
    _check(rc, "rs_adam")


def rs_adam_nvls(grad_mc: int, flag_ptrs, R: int, r: int, shard_elems: int, master, m, v, p16, *, lr, beta1, beta2, eps,
                 weight_decay, step, grad_scale, grad_f32: bool, epoch: int, counter: torch.Tensor,
                 max_blocks: int = 0, wait_seconds: float = 2.0, p16_mc: int = 0):
    """rs_adam with the gradient slice summed inside NVSwitch: grad_mc is the multicast address of the
    group's gradient buckets (candidate; the switch's summation order, not the rank order).  With
    p16_mc (multicast address of this rank's shard inside the unsharded parameter buffers) the new
    bf16 shard is stored to every rank's buffer at once and p16 is left untouched."""
    rc = lib().zb_rs_adam_nvls(c_void_p(int(grad_mc)), c_void_p(int(p16_mc)), _ptr_array(flag_ptrs), c_int(R), c_int(r), c_long(shard_elems),
                               _p(master), _p(m), _p(v), _p(p16), c_float(lr), c_float(beta1), c_float(beta2),
                               c_float(eps), c_float(weight_decay), c_int(step), c_float(grad_scale),
                               c_int(int(grad_f32)), c_int(epoch), _p(counter), c_int(max_blocks),
                               ctypes.c_double(wait_seconds), _p(status_word(master.device)), _stream())
    _check(rc, "rs_adam_nvls")


def set_rs_adam_variant(variant: int) -> None:
    """0: measured kernel; 1: candidate that requests the optimizer state and all slices up front."""
    lib().zb_set_rs_adam_variant(c_int(variant))


def wait_flags(flags: torch.Tensor, R: int, which: int, epoch: int, wait_seconds: float = 2.0):
    """One-thread kernel that returns once flags[which*R + q] >= epoch for all q (bounded)."""
    _check(lib().zb_wait_flags(_p(flags), c_int(R), c_int(which), c_int(epoch), ctypes.c_double(wait_seconds),
                               _p(status_word(flags.device)), _stream()), "wait_flags")


def peer_pull(src_ptr: int, dst: torch.Tensor, nbytes: int, max_blocks: int = 0):
    """Copies nbytes from a peer-mapped device address into dst with plain peer loads."""
    _check(lib().zb_peer_pull(c_void_p(int(src_ptr)), _p(dst), c_long(nbytes), c_int(max_blocks), _stream()),
           "peer_pull")
