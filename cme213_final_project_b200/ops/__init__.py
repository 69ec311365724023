"""Python face of the native sm_100a library (``libcme213_b200.so``, built in-tree by :mod:`.build`).

The library has a plain C ABI (pointers, sizes, a stream handle) and is loaded with ``ctypes``; every
wrapper here takes ``torch`` tensors, checks them, passes ``data_ptr()`` and the current CUDA stream, and
raises :class:`NativeError` with the library's message when a call fails.  The wrappers of the short operations do these
steps in a compiled module (``csrc/wrappers.cpp``): their calls are bound by the host.  There is no PyTorch fallback
behind these functions: on a GPU machine a missing library is an error, not a silent slow path.

The op list mirrors the reference's kernel header (``FINAL_CLEAN_CODE_/include/kernels.h:6-138``).
"""
from __future__ import annotations

import ctypes
import os
from pathlib import Path
from typing import Optional

import torch

_HERE = Path(__file__).resolve().parent
LIB_PATH = _HERE / "libcme213_b200.so"
_lib: Optional[ctypes.CDLL] = None
_tried = False

F32, BF16 = 0, 1
ACT = {"none": 0, None: 0, "relu": 1, "gelu": 2}


class NativeError(RuntimeError):
    pass


class CmeGemm(ctypes.Structure):
    _fields_ = [
        ("M", ctypes.c_int), ("N", ctypes.c_int), ("K", ctypes.c_int), ("batch", ctypes.c_int),
        ("A", ctypes.c_void_p), ("lda", ctypes.c_longlong), ("strideA", ctypes.c_longlong), ("a_trans", ctypes.c_int),
        ("B", ctypes.c_void_p), ("ldb", ctypes.c_longlong), ("strideB", ctypes.c_longlong), ("b_trans", ctypes.c_int),
        ("C", ctypes.c_void_p), ("ldc", ctypes.c_longlong), ("strideC", ctypes.c_longlong), ("c_dtype", ctypes.c_int),
        ("ab_dtype", ctypes.c_int),
        ("bias", ctypes.c_void_p),
        ("residual", ctypes.c_void_p), ("ldres", ctypes.c_longlong),
        ("aux_out", ctypes.c_void_p), ("aux_in", ctypes.c_void_p), ("ldaux", ctypes.c_longlong),
        ("act", ctypes.c_int), ("dact", ctypes.c_int), ("accumulate", ctypes.c_int),
        ("workspace", ctypes.c_void_p), ("workspace_bytes", ctypes.c_longlong),
        ("force_bn", ctypes.c_int), ("force_splits", ctypes.c_int),
        ("aux_deriv", ctypes.c_int),
        ("colsum", ctypes.c_void_p), ("colsum_slabs", ctypes.POINTER(ctypes.c_int)),
        ("allow_tf32", ctypes.c_int),
    ]


# Argument types of the entry points that are called from Python by address: with them declared, addresses and sizes go over as
# plain Python numbers (no wrapper object per argument).  v: address, i: int, l: long long, f: float, u: unsigned.
_PROTOTYPES = {
    "cme_gemm": "viv", "cme_colsum_slabs_finalize": "iviiviv", "cme_scale": "ivlfv", "cme_cast": "ivivlv",
    "cme_add": "ivvvlv", "cme_relu_bwd": "ivvvlv", "cme_init_uniform": "ivlfuv", "cme_embedding_fwd": "ivvvviiiiv",
    "cme_embedding_bwd": "ivvvviiiiiv", "cme_grad_normsq": "ivlvvv", "cme_adam": "ivvvvvlvvvffffffviv",
    "cme_copy_pair_i32": "vvvvlv", "cme_attention_fwd": "viv", "cme_attention_bwd": "viv",
}
# Entry points that the compiled wrappers call.
_WRAPPED = ("cme_last_error", "cme_cross_entropy", "cme_attention_fwd", "cme_attention_bwd", "cme_attention_path",
            "cme_attention_gemm_ws_bytes", "cme_layernorm_fwd", "cme_layernorm_bwd_blocks", "cme_layernorm_bwd",
            "cme_bias_act_residual", "cme_colsum_splits", "cme_dact_colsum", "cme_embedding_fwd", "cme_embedding_bwd")
_CTYPES = {"v": ctypes.c_void_p, "i": ctypes.c_int, "l": ctypes.c_longlong, "f": ctypes.c_float, "u": ctypes.c_uint}


def _load() -> Optional[ctypes.CDLL]:
    global _lib, _tried
    if _lib is not None or _tried:
        return _lib
    _tried = True
    if not LIB_PATH.exists():
        return None
    try:
        lib = ctypes.CDLL(str(LIB_PATH))
    except OSError:
        return None
    lib.cme_last_error.restype = ctypes.c_char_p
    lib.fnv1a_u32.restype = ctypes.c_ulonglong
    lib.fnv1a_u32.argtypes = [ctypes.c_void_p, ctypes.c_longlong, ctypes.c_ulonglong]
    lib.cme_attention_gemm_ws_bytes.restype = ctypes.c_longlong
    for name, args in _PROTOTYPES.items():
        getattr(lib, name).argtypes = [_CTYPES[c] for c in args]
    _lib = lib
    return lib


def host_lib() -> Optional[ctypes.CDLL]:
    """The library if it has been built, else ``None`` (host-only helpers have Python fallbacks)."""
    return _load()


def lib() -> ctypes.CDLL:
    l = _load()
    if l is None:
        raise NativeError(f"native library not found at {LIB_PATH}; run `python -m cme213_final_project_b200.ops.build`")
    return l


_wrappers_module = _wrappers_bound = None


def _compiled():
    """The module of compiled wrappers, for what calls no entry point of the library."""
    global _wrappers_module
    if _wrappers_module is None:
        try:
            from . import _wrappers
        except ImportError as e:
            raise NativeError(f"compiled wrappers not usable ({e}); run `python -m cme213_final_project_b200.ops.build`") from e
        _wrappers.init(NativeError)
        _wrappers_module = _wrappers
    return _wrappers_module


def _native():
    """The compiled wrappers, calling the library that :func:`lib` has loaded."""
    global _wrappers_bound
    if _wrappers_bound is None:
        l = lib()
        _wrappers = _compiled()
        _wrappers.bind(NativeError, {n: ctypes.cast(getattr(l, n), ctypes.c_void_p).value for n in _WRAPPED})
        _wrappers_bound = _wrappers
    return _wrappers_bound


def available() -> bool:
    return _load() is not None and torch.cuda.is_available()


def _check(rc: int) -> None:
    if rc != 0:
        raise NativeError(f"native call failed (status {rc}): {lib().cme_last_error().decode()}")


def _stream() -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _st() -> int:
    """The current stream's handle as a number, for the entry points with declared argument types."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _a(t: Optional[torch.Tensor]) -> Optional[int]:
    """A tensor's address as a number (likewise)."""
    return None if t is None else t.data_ptr()


_DTYPES = {torch.float32: F32, torch.bfloat16: BF16}


def _dt(t: torch.Tensor) -> int:
    d = _DTYPES.get(t.dtype)
    if d is None:
        raise NativeError(f"unsupported dtype {t.dtype}")
    return d


def _p(t: Optional[torch.Tensor]) -> ctypes.c_void_p:
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def _cuda(*ts) -> None:
    for t in ts:
        if t is not None and (not t.is_cuda or not t.is_contiguous()):
            raise NativeError("native ops need contiguous CUDA tensors")


_workspaces = {}


def workspace(nbytes: int = 64 << 20) -> torch.Tensor:
    """One fp32 scratch buffer per device that stays allocated, for callers of the C entry points who order its uses
    themselves.  ``gemm`` does not use it."""
    dev = torch.cuda.current_device()
    w = _workspaces.get(dev)
    if w is None or w.numel() * 4 < nbytes:
        w = torch.empty(nbytes // 4, dtype=torch.float32, device="cuda")
        _workspaces[dev] = w
    return w


def _scratch(device) -> Optional[torch.Tensor]:
    """64 MB for the partial sums of one product, from torch's allocator, which hands freed memory out again on the same
    stream only: products on several streams, or issued by several threads, never share it, and it goes back when the call
    has been issued.  ``None`` where there is no room: the product then runs unsplit."""
    try:
        return torch.empty(16 << 20, dtype=torch.float32, device=device)
    except torch.OutOfMemoryError:
        return None


# --------------------------------------------------------------------------------------------------
# GEMM
# --------------------------------------------------------------------------------------------------
_GEMM_BACKENDS = {"auto": 0, "tcgen05": 1, "simt": 2}


def gemm(a: torch.Tensor, b: torch.Tensor, *, a_trans: bool = False, b_trans: bool = False,
         out: Optional[torch.Tensor] = None, out_dtype: Optional[torch.dtype] = None,
         bias: Optional[torch.Tensor] = None, act: Optional[str] = None, aux_out: Optional[torch.Tensor] = None,
         dact: Optional[str] = None, aux_in: Optional[torch.Tensor] = None, residual: Optional[torch.Tensor] = None,
         accumulate: bool = False, backend: str = "auto", force_bn: int = 0, force_splits: int = 0,
         aux_deriv: bool = False, dbias: Optional[torch.Tensor] = None, allow_tf32: bool = True) -> torch.Tensor:
    """``out (+)= epilogue(op(a) @ op(b))`` for 2-D or batched 3-D row-major operands.

    ``a``: ``[M, K]`` (or ``[K, M]`` with ``a_trans``); ``b``: ``[K, N]`` (or ``[N, K]`` with ``b_trans``);
    a leading batch dimension on either operand makes the product batched (a 2-D operand is shared).
    Epilogue order: ``+bias`` -> store pre-activation to ``aux_out`` -> ``act`` -> ``* act'(aux_in)`` (``dact``)
    -> ``+residual`` -> ``+out`` (``accumulate``).  ``backend``: ``auto`` | ``tcgen05`` | ``simt``.
    ``aux_deriv``: the auxiliary tensor holds ``act'(pre-activation)`` instead of the pre-activation (forward
    stores it, backward multiplies by it).  ``dbias`` (a ``[N]`` tensor): receives the column sums of ``out`` --
    from the GEMM's own epilogue when the kernel that runs can produce them, else from a separate pass.
    fp32 operands: ``backend="simt"`` multiplies them exactly; the tcgen05 kernel takes them as tf32 (plain products
    with fp32 output only) unless ``allow_tf32=False``.  With an operand stored along M or N it takes those with K a multiple
    of four and such operands of at most 32 MB together, and ``auto`` multiplies the others exactly; ``allow_tf32=2`` lets it
    take them all.
    """
    _cuda(a, b, out, bias, aux_out, aux_in, residual, dbias)
    ws = _scratch(a.device)                           # goes back when the call has been issued
    out, part, desc = _compiled().gemm_prepare(a, b, a_trans, b_trans, out, out_dtype, bias, ACT[act], aux_out, ACT[dact], aux_in,
                                               residual, accumulate, force_bn, force_splits, aux_deriv, dbias,
                                               allow_tf32, ws)
    g = CmeGemm.from_buffer(desc)
    _check(lib().cme_gemm(ctypes.byref(g), _GEMM_BACKENDS[backend], _st()))
    if dbias is not None:
        slabs = ctypes.c_int.from_buffer(desc, ctypes.sizeof(CmeGemm)).value
        gemm.last_colsum_slabs = slabs                # 0: the epilogue did not sum (tests look at this)
        if slabs:
            _check(lib().cme_colsum_slabs_finalize(_dt(dbias), _a(part), slabs, g.N, _a(dbias), 0, _st()))
        else:
            rows = out.view(-1)[:g.batch * g.M * g.N].view(-1, g.N)
            if dbias.dtype == out.dtype:
                dact_colsum(rows, want_g=False, dbias=dbias)
            else:                                     # that pass writes the type that it reads: in fp32, then cast
                sums = dact_colsum(rows if rows.dtype == torch.float32 else cast(rows, torch.float32), want_g=False)[1]
                dbias.view(-1)[:g.N].copy_(sums)
    return out


def gemm_check_status() -> int:
    """Read and clear the device status word of the tcgen05 GEMM (non-zero: a bounded wait ran out)."""
    v = ctypes.c_int(0)
    _check(lib().cme_gemm_check_status(ctypes.byref(v)))
    return v.value


# --------------------------------------------------------------------------------------------------
# LayerNorm
# --------------------------------------------------------------------------------------------------
def layernorm_fwd(x, gamma, beta, eps: float = 1e-5, residual=None, save_sum: bool = False):
    """``y = LN(x [+ residual])``.  Returns ``(y, mean, rstd, summed)`` where ``summed`` is
    ``x + residual`` when ``save_sum`` (the fused residual + LayerNorm forward) else ``None``."""
    return _native().layernorm_fwd(x, gamma, beta, eps, residual, save_sum)


def layernorm_bwd(dy, x, gamma, mean, rstd, dres=None, dgamma=None, dbeta=None, accumulate: bool = False):
    """Returns ``(dx, dgamma, dbeta)``; ``dx`` includes ``+ dres`` when given (fused residual-gradient add)."""
    return _native().layernorm_bwd(dy, x, gamma, mean, rstd, dres, dgamma, dbeta, accumulate)


# --------------------------------------------------------------------------------------------------
# Bias / activation / residual, column sums
# --------------------------------------------------------------------------------------------------
def bias_act_residual(x, bias=None, act=None, residual=None, save_pre: bool = False):
    """``out = act(x + bias) + residual``; returns ``(out, pre)`` with ``pre = x + bias`` if ``save_pre``."""
    return _native().bias_act_residual(x, bias, ACT[act], residual, save_pre)


def dact_colsum(dout, pre=None, act=None, want_g: bool = True, dbias=None, accumulate: bool = False):
    """``g = dout * act'(pre)`` and ``dbias (+)= g.sum(0)`` — the fused activation-backward + bias-backward."""
    return _native().dact_colsum(dout, pre, ACT[act], want_g, dbias, accumulate)


def scale_(x, s: float):
    _cuda(x)
    _check(lib().cme_scale(_dt(x), _a(x), x.numel(), s, _st()))
    return x


def cast(x, dtype):
    _cuda(x)
    y = torch.empty(x.shape, dtype=dtype, device=x.device)
    _check(lib().cme_cast(_dt(x), _a(x), _dt(y), _a(y), x.numel(), _st()))
    return y


def add(a, b):
    _cuda(a, b)
    out = torch.empty_like(a)
    _check(lib().cme_add(_dt(a), _a(a), _a(b), _a(out), a.numel(), _st()))
    return out


def relu_bwd(x, dy):
    _cuda(x, dy)
    dx = torch.empty_like(dy)
    _check(lib().cme_relu_bwd(_dt(x), _a(x), _a(dy), _a(dx), x.numel(), _st()))
    return dx


def init_uniform_(out, scale: float, seed: int):
    _cuda(out)
    _check(lib().cme_init_uniform(_dt(out), _a(out), out.numel(), scale, seed & 0xFFFFFFFF, _st()))
    return out


# --------------------------------------------------------------------------------------------------
# Embedding
# --------------------------------------------------------------------------------------------------
def embedding_fwd(tokens, tok, pos):
    return _native().embedding_fwd(tokens, tok, pos)


def embedding_bwd(tokens, dout, V: int, T: int, dtok=None, dpos=None, accumulate: bool = False):
    return _native().embedding_bwd(tokens, dout, V, T, dtok, dpos, accumulate)


# --------------------------------------------------------------------------------------------------
# Loss and optimizer
# --------------------------------------------------------------------------------------------------
def cross_entropy(logits, targets, grad_scale: Optional[float] = None, prob_eps: float = 0.0, inplace: bool = False):
    """Returns ``(mean loss [1] fp32, dlogits, per-row losses)``; ``dlogits = (softmax - onehot) * grad_scale``
    (default ``1/rows``).  ``prob_eps = 1e-9`` reproduces the reference's ``-log(p + 1e-9)`` form."""
    return _native().cross_entropy(logits, targets, grad_scale, prob_eps, inplace)


def grad_normsq(g):
    _cuda(g)
    partial = torch.empty(1024, dtype=torch.float32, device=g.device)
    out = torch.empty(1, dtype=torch.float32, device=g.device)
    _check(lib().cme_grad_normsq(_dt(g), _a(g), g.numel(), _a(partial), _a(out), _st()))
    return out


def adam_step(master, grads, m, v, step_dev, lr_dev, *, compute=None, normsq=None, beta1=0.9, beta2=0.999, eps=1e-8,
              weight_decay=0.0, grad_scale=1.0, clip_norm=0.0, nodecay=None):
    """One Adam / AdamW update over a flat range.  ``step_dev`` (int32 [1], already incremented) and
    ``lr_dev`` (fp32 [1]) live on the device; ``nodecay`` is an int64 ``[k, 2]`` tensor of sorted ranges."""
    _cuda(master, grads, m, v, step_dev, lr_dev, compute, normsq, nodecay)
    nn = 0 if nodecay is None else nodecay.shape[0]
    _check(lib().cme_adam(_dt(grads), _a(master), _a(compute), _a(grads), _a(m), _a(v), master.numel(),
                          _a(step_dev), _a(lr_dev), _a(normsq), beta1, beta2, eps, weight_decay, grad_scale, clip_norm,
                          _a(nodecay), nn, _st()))


# --------------------------------------------------------------------------------------------------
# Attention
# --------------------------------------------------------------------------------------------------
class CmeAttn(ctypes.Structure):
    _fields_ = [
        ("nb", ctypes.c_int), ("nh", ctypes.c_int), ("T", ctypes.c_int), ("HD", ctypes.c_int),
        ("sb", ctypes.c_longlong), ("sh", ctypes.c_longlong), ("st", ctypes.c_longlong),
        ("osb", ctypes.c_longlong), ("osh", ctypes.c_longlong), ("ost", ctypes.c_longlong),
        ("causal", ctypes.c_int), ("scale", ctypes.c_float), ("dtype", ctypes.c_int),
        ("q", ctypes.c_void_p), ("k", ctypes.c_void_p), ("v", ctypes.c_void_p), ("o", ctypes.c_void_p),
        ("lse", ctypes.c_void_p),
        ("d_o", ctypes.c_void_p), ("dq", ctypes.c_void_p), ("dk", ctypes.c_void_p), ("dv", ctypes.c_void_p),
        ("delta", ctypes.c_void_p), ("dq_accum", ctypes.c_void_p),
        ("ws", ctypes.c_void_p), ("ws_bytes", ctypes.c_longlong),
        ("dq_sem", ctypes.c_void_p), ("dq_mode", ctypes.c_int), ("dq_accum_clean", ctypes.c_int),
    ]


_BACKENDS = {"auto": 0, "tc": 1, "simt": 2, "gemm": 3}


def _attn_desc(q, B, H, T, layout, causal):
    """The descriptor for those who call the C entry points themselves, with strides and buffers of their own; ``attention_fwd`` and
    ``attention_bwd`` fill theirs in compiled code."""
    D = q.shape[-1]
    HD = D // H
    nb, nh, sb, sh, st = (B * H, 1, T * HD, 0, HD) if layout == "flat" else (B, H, T * D, HD, D)
    a = CmeAttn(nb, nh, T, HD, sb, sh, st, sb, sh, st, int(causal), 1.0 / (HD ** 0.5), _dt(q))
    if layout == "flat" and T <= 512 and q.dtype == torch.bfloat16:      # scratch of the batched-GEMM path
        nbytes = int(lib().cme_attention_gemm_ws_bytes(B * H, T))
        ws = torch.empty(nbytes + 256, dtype=torch.uint8, device=q.device)
        a._ws_keepalive = ws
        a.ws = (ws.data_ptr() + 255) // 256 * 256
        a.ws_bytes = nbytes
    return a


def attention_fwd(q, k, v, B: int, H: int, T: int, layout: str = "split", causal: bool = False,
                  backend: str = "auto"):
    """``q, k, v``: ``[B*T, D]``.  ``layout="flat"`` views each as ``[B*H, T, HD]`` without a transpose (the
    reference's head layout); ``"split"`` is the standard ``[B, T, H, HD]`` split.  Returns ``(out, lse)``."""
    return _native().attention_fwd(q, k, v, B, H, T, layout == "flat", int(causal), _BACKENDS[backend])


def attention_bwd(q, k, v, out, lse, dout, B: int, H: int, T: int, layout: str = "split", causal: bool = False,
                  backend: str = "auto", ordered_dq: bool = False, dq_mode: Optional[int] = None,
                  scratch=None):
    """Returns ``(dq, dk, dv)``.  How the tensor-core kernel completes dQ from the key blocks' parts (``dq_mode``):
    0 (default) clears an fp32 scratch, adds the parts in arrival order and converts the sums with a second kernel;
    1 (``ordered_dq``) adds them in a fixed order (bit-reproducible, slower); 2 (up to 64 query blocks) adds them in
    arrival order and lets the CTA whose part comes last scale and cast the sums (two launches fewer, slower at
    large shapes).  ``scratch`` = (fp32 tensor of ``q.numel()``
    zeros, int32 tensor of ``B * H * ceil(T / 128)`` zeros) lets calls share the buffers; modes 1 and 2 leave both
    zero again."""
    if dq_mode is None:
        dq_mode = 1 if ordered_dq else 0
    acc, sem = (None, None) if scratch is None else scratch
    return _native().attention_bwd(q, k, v, out, lse, dout, B, H, T, layout == "flat", int(causal), _BACKENDS[backend], int(dq_mode),
                                   acc, sem)


def launch_count() -> int:
    """Kernels launched (or captured) by the native library so far in this process."""
    l = lib()
    l.cme_launch_count.restype = ctypes.c_longlong
    return int(l.cme_launch_count())


def attention_check_status() -> int:
    """Read and clear the status word of the tensor-core attention kernels (non-zero: a wait ran out)."""
    v = ctypes.c_int(0)
    _check(lib().cme_attention_check_status(ctypes.byref(v)))
    return v.value
