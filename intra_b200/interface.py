"""Python entry points, drop-in for the reference's `intra_attn/interface.py`.

Same names, defaults, argument meaning and exceptions as the reference
(intra_attn/interface.py:17-66); the work is done by libintra_b200.so through its C ABI.
All functions take q, k, v of shape (batch, seqlen, heads, 128) in bfloat16 on a B200 and return the
attention output shaped, typed and laid out like q. k/v may have fewer heads than q (GQA) as long as
they divide the query heads. Forward only.
"""
from __future__ import annotations

import ctypes
import numbers

import torch

from . import _loader
from ._loader import lib

LLM_PATTERNS = {"scatter": 0, "gather1": 1, "window": 4}
IMAGE_PATTERNS = {"scatter": 0, "gather0": 4}
TEXT_LEN = 512


def _torch_name(path):
    """torch.<path>, or None where this release of torch has no such name."""
    obj = torch
    for part in path.split("."):
        obj = getattr(obj, part, None)
    return obj


# What torch keeps under private names: the current stream's handle, and whatever looks inside operators.
_raw_stream = _torch_name("_C._cuda_getCurrentRawStream") or (lambda index: torch.cuda.current_stream(index).cuda_stream)
_tracing_state = _torch_name("_C._get_tracing_state")
_dispatch_modes = _torch_name("_C._len_torch_dispatch_stack")
_functorch_level = _torch_name("_C._functorch.peek_interpreter_stack")
_forward_ad = _torch_name("autograd.forward_ad")
_function_modes = _torch_name("_C._len_torch_function_stack")
_function_mode_stack = _torch_name("overrides._get_current_function_mode_stack")
try:
    from torch.utils._device import DeviceContext as _device_context
except ImportError:
    _device_context = None


def _watched():
    """Does something look at the operators that are called now: tracing, a dispatch or function mode, vmap and its like,
    forward-mode? True, too, where this release of torch does not tell. A default device is a function mode that only
    places new tensors."""
    if _tracing_state is None or _dispatch_modes is None or _functorch_level is None or _function_modes is None:
        return True
    if _function_modes() > 0 and (_function_mode_stack is None or any(type(m) is not _device_context for m in _function_mode_stack())):
        return True
    return (_tracing_state() is not None or _dispatch_modes() > 0 or _functorch_level() is not None
            or getattr(_forward_ad, "_current_level", 0) >= 0)


def _check(q, k, v):
    """Argument checks of the reference (intra_attn/interface.py:17-23), plus the layout the
    library needs: the reference's kernels silently assume 128-element head stride and equal q/k row
    strides; here any batch/token/head strides are honoured as long as rows stay 16-byte aligned,
    and tensors that break that are made contiguous first."""
    for x in (q, k, v):
        if not x.is_cuda or x.dtype != torch.bfloat16 or x.shape[-1] != 128:
            raise ValueError("INTRA kernels need CUDA bfloat16 tensors with head_dim 128")
    if torch.is_grad_enabled() and any(x.requires_grad for x in (q, k, v)):
        raise RuntimeError("INTRA kernels are forward-only; call them under torch.no_grad()")
    if q.dim() != 4 or k.dim() != 4 or v.dim() != 4:
        raise ValueError("q, k, v must be (batch, seqlen, heads, 128)")
    if k.shape != v.shape or k.shape[:2] != q.shape[:2] or q.shape[2] % k.shape[2] != 0:
        raise ValueError(f"incompatible shapes q={tuple(q.shape)} k={tuple(k.shape)} v={tuple(v.shape)}")
    if k.device != q.device or v.device != q.device:
        raise ValueError("q, k, v must be on the same device")

    def usable(x):
        return (x.stride(-1) == 1 and x.data_ptr() % 16 == 0
                and all(x.stride(d) % 8 == 0 and x.stride(d) >= 0 for d in range(3)))

    return [x if usable(x) else x.contiguous() for x in (q, k, v)]


def _scale(q, softmax_scale):
    return q.shape[-1] ** -0.5 if softmax_scale is None else float(softmax_scale)


def _raise(status):
    msg = _loader.strerror(status)
    if status == _loader.ERR_CUDA:
        raise RuntimeError(f"intra_b200: {msg} (cudaError {lib.intra_b200_last_cuda_error()})")
    if status in (_loader.ERR_DEVICE, _loader.ERR_KERNEL):
        raise RuntimeError(f"intra_b200: {msg}")
    raise ValueError(f"intra_b200: {msg}")


def _byte_span(x):
    """[first, last) byte addresses a tensor with non-negative strides can touch."""
    last = sum((n - 1) * st for n, st in zip(x.shape, x.stride()) if n > 0)
    return x.data_ptr(), x.data_ptr() + (last + 1) * x.element_size()


def _check_out(out, q, inputs):
    """Checks of a caller's output tensor, (B, S, H, 128) like q."""
    if out.shape != q.shape or out.dtype != q.dtype or out.device != q.device:
        raise ValueError("out must match q in shape, dtype and device")
    if out.stride(-1) != 1 or any(out.stride(d) % 8 or out.stride(d) <= 0 for d in range(3)) or out.data_ptr() % 16:
        raise ValueError("out needs unit stride in the last dim, positive strides and 16-byte aligned rows")
    lo, hi = _byte_span(out)
    for x in inputs:
        xlo, xhi = _byte_span(x)
        if lo < xhi and xlo < hi:
            raise ValueError("out must not overlap q, k or v: other tiles still read them while it is written")


# int64[3] constants for the C ABI by their values: building one costs as much as a tenth of a short call.
_STRIDES = {}
_STRIDES_MAX = 1024


def _c_strides(batch, token, head):
    key = (batch, token, head)
    arr = _STRIDES.get(key)
    if arr is None:
        if len(_STRIDES) >= _STRIDES_MAX:
            _STRIDES.clear()
        arr = _STRIDES[key] = (ctypes.c_int64 * 3)(batch, token, head)
    return arr


def _prepare(q, k, v, token, head, out):
    """Checks and output of a call whose q, k, v have their token and head axes at `token` and `head` (1 and 2, or
    2 and 1). Returns (data pointers of q, k, v and the output, B, S, H, Hkv, their strides for the C ABI, the output
    as (B, S, H, 128), and the tensors read, copies perhaps, to be held until the launch). What this function's own tests do not recognise at once goes through `_check`, which raises
    or copies. Nothing is remembered about tensors."""
    if (q.requires_grad or k.requires_grad or v.requires_grad) and torch.is_grad_enabled():
        raise RuntimeError("INTRA kernels are forward-only; call them under torch.no_grad()")
    bf16 = torch.bfloat16
    qn, kn = q.shape, k.shape
    ready = False
    if (q.is_cuda and k.is_cuda and v.is_cuda and q.dtype is bf16 and k.dtype is bf16 and v.dtype is bf16
            and len(qn) == 4 and len(kn) == 4 and kn == v.shape and qn[3] == 128 and kn[3] == 128 and qn[0] == kn[0]
            and qn[token] == kn[token] and kn[head] > 0 and qn[head] % kn[head] == 0
            and k.device == q.device and v.device == q.device):
        qs, ks, vs = q.stride(), k.stride(), v.stride()
        ptrs = q.data_ptr(), k.data_ptr(), v.data_ptr()
        ready = (qs[3] == 1 and ks[3] == 1 and vs[3] == 1 and not (ptrs[0] | ptrs[1] | ptrs[2]) & 15
                 and not (qs[0] | qs[1] | qs[2] | ks[0] | ks[1] | ks[2] | vs[0] | vs[1] | vs[2]) & 7)
    if not ready:
        if token == 2:
            q, k, v = q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2)
            token, head = 1, 2
        q, k, v = _check(q, k, v)
        qn, kn = q.shape, k.shape
        qs, ks, vs = q.stride(), k.stride(), v.stride()
        ptrs = q.data_ptr(), k.data_ptr(), v.data_ptr()
    if out is not None:
        _check_out(out, q, (q, k, v))                # only calls in (B, S, H, 128) order take `out`
        os_ = out.stride()
        optr = out.data_ptr()
    else:
        out = torch.empty_like(q)
        os_ = out.stride()
        if os_[3] != 1 or (os_[0] | os_[1] | os_[2]) & 7 or os_[0] <= 0 or os_[1] <= 0 or os_[2] <= 0:
            out = torch.empty((qn[0], qn[token], qn[head], 128), dtype=bf16, device=q.device)
            if token == 2:
                out = out.transpose(1, 2)
            os_ = out.stride()
        optr = out.data_ptr()
        if token == 2:
            out = out.transpose(1, 2)
    return (ptrs[0], ptrs[1], ptrs[2], optr, qn[0], qn[token], qn[head], kn[head],
            _c_strides(qs[0], qs[token], qs[head]), _c_strides(ks[0], ks[token], ks[head]),
            _c_strides(vs[0], vs[token], vs[head]), _c_strides(os_[0], os_[token], os_[head]), out, (q, k, v))


def _llm(q, k, v, token, head, pattern, group_num, window, softmax_scale, strict, return_lse, out):
    qp, kp, vp, op, B, S, H, Hkv, qs, ks, vs, os_, out, held = _prepare(q, k, v, token, head, out)
    if strict and pattern == "gather1" and (group_num != 8 or S % (group_num * group_num)):
        raise ValueError(f"gather1 needs group_num=8 and seqlen % 64 == 0, got G={group_num}, S={S}")
    pid = LLM_PATTERNS[pattern]
    dev = out.device
    tail = (qs, ks, vs, os_, pid, int(group_num), int(window), _scale(out, softmax_scale), dev.index,
            _raw_stream(dev.index))
    if return_lse:
        lse = torch.empty((B, H, S), dtype=torch.float32, device=dev)
        rc = lib.intra_b200_fwd_llm_lse(qp, kp, vp, op, lse.data_ptr(), B, S, H, Hkv, *tail)
    else:
        rc = lib.intra_b200_fwd_llm(qp, kp, vp, op, B, S, H, Hkv, *tail)
    if rc != 0:
        _raise(rc)
    return (out, lse) if return_lse else out


def _image(q, k, v, token, head, pattern, width, softmax_scale, strict, return_lse, out):
    qp, kp, vp, op, B, S, H, Hkv, qs, ks, vs, os_, out, held = _prepare(q, k, v, token, head, out)
    if not strict and (width < 16 or width % 8):
        raise ValueError("width must be a multiple of 8 and at least 16")
    if strict and width not in (64, 128):
        raise ValueError("image kernels are compiled for width 64 and 128")
    if S != TEXT_LEN + width * width:
        raise ValueError(f"expected {TEXT_LEN} text + {width}x{width} image tokens, got {S}")
    if Hkv != H:
        raise ValueError("image attention is multi-head: k/v need as many heads as q")
    pid = IMAGE_PATTERNS[pattern]
    dev = out.device
    tail = (qs, ks, vs, os_, pid, int(width), _scale(out, softmax_scale), dev.index,
            _raw_stream(dev.index))
    if return_lse:
        lse = torch.empty((B, H, S), dtype=torch.float32, device=dev)
        rc = lib.intra_b200_fwd_image_lse(qp, kp, vp, op, lse.data_ptr(), B, S, H, *tail)
    else:
        rc = lib.intra_b200_fwd_image(qp, kp, vp, op, B, S, H, *tail)
    if rc != 0:
        _raise(rc)
    return (out, lse) if return_lse else out


def intra_llm_attn(q, k, v, pattern="scatter", group_num=8, window=576, softmax_scale=None, *, strict=True,
                   return_lse=False, out=None):
    """Causal prefill attention for language models.

    pattern="scatter": token i attends to earlier tokens j with j % group_num == i % group_num.
    pattern="gather1": groups are segments of group_num tokens, segment s in group s % group_num.
    pattern="window":  each 64-query block attends to itself and the preceding window - 64 tokens.

    Any seqlen works for scatter and window; gather1 keeps the reference's contract of
    group_num=8 and seqlen % 64 == 0 (intra_attn/interface.py:41-42). `strict=False` (not in the
    reference) lifts that restriction: the kernels handle Gather-1 for any group_num and seqlen.
    `return_lse=True` (not in the reference, whose kernels compute the value and drop it) returns
    `(out, lse)` with lse of shape (batch, heads, seqlen), float32: the log of each query's softmax
    denominator, which is what merging attention over disjoint key sets needs. `out=` (not in the
    reference, which always allocates) writes into a tensor of the caller's; it must not alias q, k, v.
    """
    return _llm(q, k, v, 1, 2, pattern, group_num, window, softmax_scale, strict, return_lse, out)


def intra_image_attn(q, k, v, pattern="scatter", width=64, softmax_scale=None, *, strict=True, return_lse=False,
                     out=None):
    """Bidirectional attention for FLUX-style sequences: 512 text tokens followed by a
    width x width grid of image tokens.

    pattern="scatter": 8 groups, image token (r, c) in group (r % 2) * 4 + c % 4; text chunks of
                       64 tokens ride with groups 0..7; all text keys are always visible.
    pattern="gather0": each 8 x 8 image patch attends to a 16 x 16 window around it plus all text.

    width must be 64 or 128 as in the reference (intra_attn/interface.py:60-63); `strict=False` (not in
    the reference) accepts any width that is a multiple of 8 and at least 16. `return_lse=True` returns
    `(out, lse)` and `out=` writes into the caller's tensor, as in intra_llm_attn.
    """
    return _image(q, k, v, 1, 2, pattern, width, softmax_scale, strict, return_lse, out)


def decode_attn(q, k, v, mask=None, softmax_scale=None):
    """Dense attention of one token per sequence over its cache: q (B, H, 1, 128), k and v
    (B, Hkv, S, 128), `mask` None or bool (B or 1, 1, 1, >= S), nonzero = visible. Returns (B, 1, H, 128), or None
    for calls the decode kernel does not take - other types, GPUs, layouts or broadcasts, masks per
    head or additive, and everything that looks inside an operator (autograd, forward-mode, vmap, tracing,
    dispatch modes, autocast to another type) - which are the caller's to run as torch operators."""
    # what costs least first, tracers before sizes: a call that is left to torch has paid for the questions before it
    if type(q) is not torch.Tensor or type(k) is not torch.Tensor or type(v) is not torch.Tensor:
        return None
    if q.dtype != torch.bfloat16 or k.dtype != torch.bfloat16 or v.dtype != torch.bfloat16 or not q.is_cuda:
        return None
    if mask is not None and (type(mask) is not torch.Tensor or mask.dtype != torch.bool or mask.dim() != 4):
        return None
    if torch.compiler.is_compiling() or _watched():
        return None
    kn = k.shape
    if q.dim() != 4 or len(kn) != 4 or kn != v.shape:
        return None
    B, H, n, D = q.shape
    Bk, Hkv, S, Dk = kn
    if n != 1 or D != 128 or Dk != 128 or Bk != B or B == 0 or S == 0 or Hkv == 0 or H < Hkv or H % Hkv:
        return None
    if torch.is_grad_enabled() and (q.requires_grad or k.requires_grad or v.requires_grad):
        return None
    if softmax_scale is not None and type(softmax_scale) is not float and not isinstance(softmax_scale, numbers.Real):
        return None
    dev = q.device
    if (q.is_neg() or k.is_neg() or v.is_neg() or k.device != dev or v.device != dev
            or (torch.is_autocast_enabled("cuda") and torch.get_autocast_dtype("cuda") != torch.bfloat16)):
        return None
    qs, ks, vs = q.stride(), k.stride(), v.stride()
    qp, kp, vp = q.data_ptr(), k.data_ptr(), v.data_ptr()
    if (qs[3] != 1 or ks[3] != 1 or vs[3] != 1 or (qp | kp | vp) & 15
            or (qs[0] | qs[1] | ks[0] | ks[1] | ks[2] | vs[0] | vs[1] | vs[2]) & 7):
        return None
    mp, ms0, ms1 = None, 0, 0
    if mask is not None:
        if mask.device != dev or mask.shape[0] not in (1, B) or mask.shape[1] != 1 or mask.shape[2] != 1 or mask.shape[3] < S:
            return None
        mp, ms0, ms1 = mask.data_ptr(), mask.stride(0) if mask.shape[0] == B else 0, mask.stride(3)
    out = q.new_empty((B, 1, H, D))
    need = ctypes.c_int64(0)
    scratch, nbytes = None, 0
    while True:
        rc = lib.intra_b200_decode(qp, kp, vp, mp, out.data_ptr(), None if scratch is None else scratch.data_ptr(), nbytes,
                                   need, B, S, H, Hkv, qs[0], qs[1], ks[0], ks[2], ks[1], vs[0], vs[2], vs[1], ms0, ms1,
                                   0.08838834764831845 if softmax_scale is None else softmax_scale, dev.index,
                                   _raw_stream(dev.index))
        if rc != _loader.NEED_SCRATCH:
            break
        nbytes = need.value
        scratch = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    if rc == _loader.ERR_DEVICE:                     # another GPU than the kernels are built for
        return None
    if rc != 0:
        _raise(rc)
    return out


def device_status(device=None, reset=False):
    """Synchronise `device` and return the status word its kernels write when a bounded wait gives
    up (0 = healthy; otherwise 100 + the id of the first wait that ran out since the last reset). The
    attention calls never poll it, and a recorded failure does not change later launches: a caller that
    wants to know checks here, e.g. once per step. Raises nothing; callers decide."""
    dev = torch.cuda.current_device() if device is None else torch.device(device).index
    word = ctypes.c_int(0)
    lib.intra_b200_device_status(dev, ctypes.byref(word), 1 if reset else 0)
    return word.value
